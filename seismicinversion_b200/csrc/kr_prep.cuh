// Per-slowness preparation of the derivative kernels: layer terms and derivative factors,
// interface coefficients and their tangents.
#pragma once

#include "kr_adjoint.cuh"
#include "kr_internal.cuh"

namespace kr {

// One block per (slowness, chunk of kPrepThreads interface items): the layer terms and
// derivative factors of the chunk's layers go to shared memory, then one thread per
// (interface, item): items 0..5 form one tangent column each, item 6 the interface's
// coefficients and the workspace copy of its upper layer (and of the half-space, for the last
// interface), so no lane of a warp waits on another's extra work.  The coefficients read the
// layer terms back from shared memory after a barrier, as the forward kernel's prologue
// does, so they round exactly as there.  Blocks of 128 threads:
// with 64, twice as many SMs are busy with 250 registers a thread while the frequency-sum sweep
// runs beside this kernel (64 x 32 gradient 65 us against 56), and kernels that wait for it gain
// nothing (64 x 1024 Jacobian 106.4 against 106.2).
constexpr int kPrepThreads = 128;
constexpr int kPrepItems = 7;                               // per interface
constexpr int kPrepLayers = kPrepThreads / kPrepItems + 3;  // layers one chunk touches

static __global__ void __launch_bounds__(kPrepThreads)
deriv_prep_kernel(const double* __restrict__ tab, int L, const double* __restrict__ p,
                  int n_chunks, LayerP* lay, LayerD* dlay, Iface* coef, ScatTan* tan) {
  // a sweep that forms its own coefficients may start at once (it waits for this grid before it
  // reads the tangents)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ LayerP s_lp[kPrepLayers];
  __shared__ LayerD s_ld[kPrepLayers];
  const int I = L - 1;
  const int j = blockIdx.x / n_chunks;
  const int t0 = (blockIdx.x % n_chunks) * kPrepThreads;
  const int t1 = min(t0 + kPrepThreads, kPrepItems * I);
  const int l0 = t0 / kPrepItems, l1 = (t1 - 1) / kPrepItems + 1;  // the chunk's layers
  const double pj = p[j];
  for (int l = l0 + threadIdx.x; l <= l1; l += blockDim.x) {
    const LayerP lp = layer_terms(tab, L, l, pj);
    s_lp[l - l0] = lp;
    s_ld[l - l0] = layer_derivs(tab, L, l, pj, lp);
  }
  __syncthreads();
  const int t = t0 + threadIdx.x;
  if (t >= t1) return;
  const int i = t / kPrepItems, item = t % kPrepItems;
  const size_t idx = (size_t)j * I + i, e = (size_t)j * L + i;
  const LayerP& up = s_lp[i - l0];
  const LayerP& lo = s_lp[i + 1 - l0];
  if (item == 6) {
    lay[e] = up;
    dlay[e] = s_ld[i - l0];
    if (i == I - 1) {
      lay[e + 1] = lo;
      dlay[e + 1] = s_ld[i + 1 - l0];
    }
    coef[idx] = interface_coeffs(pj, i, up, lo);
    return;
  }
  cd c[10];
  interface_tangent_col(pj, i, up, s_ld[i - l0], lo, s_ld[i + 1 - l0], item, c);
  for (int k = 0; k < 10; ++k) tan[idx].t[k][item] = c[k];
}

static kr_status launch_prep(const double* layers, int L, const double* p, int n_p, LayerP* lay,
                             LayerD* dlay, Iface* coef, ScatTan* tan, cudaStream_t st,
                             const char* what) {
  const int n_chunks = (kPrepItems * (L - 1) + kPrepThreads - 1) / kPrepThreads;
  if ((size_t)n_p * n_chunks > 0x7fffffffULL) return KR_ERR_TOO_LARGE;
  deriv_prep_kernel<<<(unsigned)(n_p * n_chunks), kPrepThreads, 0, st>>>(layers, L, p, n_chunks, lay,
                                                                         dlay, coef, tan);
  return check_launch(what);
}

}  // namespace kr
