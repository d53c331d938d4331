// Internal declarations shared by the library's translation units (not part of the C-ABI).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <mutex>

#include "../../include/kennett_b200.h"
#include "kr_math.cuh"

namespace kr {

constexpr int kMaxLayers = KR_MAX_LAYERS;

// Dynamic shared memory of the per-slowness prologue: layer terms + interface coefficients.
__host__ __device__ inline size_t prologue_smem_bytes(int n_layers) {
  return sizeof(LayerP) * (size_t)n_layers + sizeof(Iface) * (size_t)(n_layers - 1);
}

inline kr_status cuda_status(cudaError_t e) { return e == cudaSuccess ? KR_OK : KR_ERR_CUDA; }

// Complex arrays are read and written as 16-byte units (vector loads, cp.async): every
// complex pointer of the C ABI must be 16-byte aligned.  Null passes (checked separately).
inline bool aligned16(const void* ptr) { return ((uintptr_t)ptr & 15u) == 0; }

// Remembers the last CUDA error string for kr_last_error().
void set_last_error(const char* where, cudaError_t e);
void set_last_error_msg(const char* msg);

// Raises a kernel's dynamic shared-memory limit to `bytes` on the current device, calling the
// runtime only when the limit recorded for that device is lower: after the first call per
// device (and larger size) a launcher makes no runtime call but the launch, so it can be
// captured into a CUDA graph.  `lim` is the launcher's own per-kernel table (zero-initialised
// static storage).
constexpr int kMaxDevices = 64;
struct SmemLimit {
  int bytes[kMaxDevices];
};
// One lock for every kernel's limit: host threads that launch concurrently (two servers, a
// server and a direct call) must not interleave the check, the attribute call and the
// record, or one could lower a limit another thread's launch relies on.  Under the lock a
// limit only ever rises.
inline std::mutex& smem_limit_mutex() {
  static std::mutex m;
  return m;
}

inline kr_status raise_smem_limit(const void* fn, size_t bytes, SmemLimit& lim,
                                  const char* where) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_last_error(where, e);
    return KR_ERR_CUDA;
  }
  const bool known = dev >= 0 && dev < kMaxDevices;
  std::lock_guard<std::mutex> g(smem_limit_mutex());
  if (known && lim.bytes[dev] >= (int)bytes) return KR_OK;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) {
    set_last_error(where, e);
    return KR_ERR_CUDA;
  }
  if (known) lim.bytes[dev] = (int)bytes;
  return KR_OK;
}

inline kr_status check_launch(const char* where) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_error(where, e);
    return KR_ERR_CUDA;
  }
  return KR_OK;
}

// Block-cooperative copy of n bytes (multiple of 16, 16-byte aligned) into shared memory.
__device__ __forceinline__ void copy16(void* dst, const void* src, size_t n) {
  double2* d = reinterpret_cast<double2*>(dst);
  const double2* s = reinterpret_cast<const double2*>(src);
  for (size_t k = threadIdx.x; k < n / 16; k += blockDim.x) d[k] = s[k];
}

}  // namespace kr
