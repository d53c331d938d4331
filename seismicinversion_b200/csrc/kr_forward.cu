// Fused forward reflectivity kernel: R[p][omega] of one model.
//
// kr_forward.cuh's kernel with the Kennett recursion: the cumulative reflection matrix in
// registers.  FP64 CUDA cores; no tensor-core work exists here (2x2 complex algebra per thread is
// not a contraction).
//
// The bound is the FP64 pipe fed by the register file: an FMA with three distinct register
// operands issues at 13.5e12 / s on this GPU (two operands: 18e12), and the 21-layer
// 8192 x 2047 grid runs at 12.9e12 (119 FP64 instructions per update, 3.1 ms; the form with
// two phases per step, a correctly rounded division and a block per slowness took 132 and
// 3.3 ms).  4096 x 2047 slownesses of a 5-layer model: 389 -> 322 us; 2048 x 511: 137 -> 58 us
// (several slownesses share a prologue); 193 x 1501 of a 64-layer model: 351 -> 230 us (table
// instead of direct exponentials).  Two frequencies per lane (half the coefficient loads, two
// chains) measured the same on 21 layers and 7 % slower on 5: registers, not loads, bound it.
#include <stdlib.h>

#include "kr_forward.cuh"

namespace kr {

// Register budget of the three-phase kernel: blocks of 128 threads resident per SM the compiler
// must allow (4 -> 128 registers, 5 -> 96, 6 -> 80).  Set by kr_set_forward_variant or the
// KR_FWD_MINB environment variable; otherwise 4 (5-layer grid: 322 us at 4, 359 at 5, 363 at 6;
// 30 layers: 645, 695, 713).
static int g_fwd_minb = -1;  // -1: not read yet, 0: automatic

static int forward_minb() {
  if (g_fwd_minb < 0) {
    const char* e = getenv("KR_FWD_MINB");
    const int v = e ? atoi(e) : 0;
    g_fwd_minb = (v >= 4 && v <= 6) ? v : 0;
  }
  return g_fwd_minb > 0 ? g_fwd_minb : 4;
}

}  // namespace kr

using namespace kr;

extern "C" void kr_set_forward_variant(int32_t min_blocks_per_sm) {
  g_fwd_minb = (min_blocks_per_sm >= 4 && min_blocks_per_sm <= 6) ? min_blocks_per_sm : 0;
}

extern "C" kr_status kr_reflectivity(const double* layers, int32_t n_layers, const double* p,
                                     int32_t n_p, const double* omega, int32_t n_w,
                                     uint32_t flags, double* R, void* stream) {
  if (n_p < 0 || n_w < 0 || (flags & ~KR_FREE_SURFACE)) return KR_ERR_INVALID_ARGUMENT;
  if (n_layers < 2) return KR_ERR_INVALID_MODEL;
  if (n_layers > kMaxLayers) return KR_ERR_TOO_LARGE;
  if (n_p == 0 || n_w == 0) return KR_OK;
  if (!layers || !p || !omega || !R) return KR_ERR_INVALID_ARGUMENT;
  if (!aligned16(omega) || !aligned16(R)) return KR_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  constexpr const char* kWhat = "kr_reflectivity";
  if (n_layers > kPqsLayers)
    return launch_forward_deep<KennettForm>(kWhat, layers, n_layers, p, n_p, omega, n_w, flags, R, st);
  switch (forward_minb()) {
    case 6:
      return launch_forward<KennettForm, 3, 1, 4, 6>(kWhat, layers, n_layers, p, n_p, omega, n_w, flags, R, st);
    case 5:
      return launch_forward<KennettForm, 3, 1, 4, 5>(kWhat, layers, n_layers, p, n_p, omega, n_w, flags, R, st);
    default:
      return launch_forward<KennettForm, 3, 1, 4, 4>(kWhat, layers, n_layers, p, n_p, omega, n_w, flags, R, st);
  }
}
