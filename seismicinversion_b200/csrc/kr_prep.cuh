// Per-slowness preparation of the derivative kernels: layer terms and derivative factors,
// interface coefficients and their tangents.
#pragma once

#include "kr_adjoint.cuh"
#include "kr_internal.cuh"

namespace kr {

// One thread per (slowness, interface, item), blocks of kPrepThreads of them in that order: the layer
// terms and derivative factors of the layers a block touches go to shared memory, then items 0..5
// form one tangent column each, item 6 the interface's coefficients and the workspace copy of its
// upper layer (and of the half-space, for the last interface), so no lane of a warp waits on
// another's extra work.  The coefficients read the layer terms back from shared memory after a
// barrier, as the forward kernel's prologue does, so they round exactly as there.  A block takes as
// many slownesses as its threads hold: with chunks of one slowness a 3-layer model kept 14 of 128
// threads busy (gradient of 2000 slownesses x 128 frequencies 119 us against 56) and one of 21 layers
// left a second block nearly empty, which kept the sweep's blocks waiting (64 x 128: 59 against 36).
// Blocks of 128 threads:
// with 64, twice as many SMs are busy with 250 registers a thread while the frequency-sum sweep
// runs beside this kernel (64 x 32 gradient 65 us against 56), and kernels that wait for it gain
// nothing (64 x 1024 Jacobian 106.4 against 106.2).
constexpr int kPrepThreads = 128;
constexpr int kPrepItems = 7;  // per interface
// Interfaces a block touches, and layers: each interface's upper one, and each slowness's last.
constexpr int kPrepIfaces = kPrepThreads / kPrepItems + 2;
constexpr int kPrepLayers = 2 * kPrepIfaces;

static __global__ void __launch_bounds__(kPrepThreads)
deriv_prep_kernel(const double* __restrict__ tab, int L, const double* __restrict__ p,
                  unsigned n_items, LayerP* lay, LayerD* dlay, Iface* coef, ScatTan* tan) {
  // a sweep that forms its own coefficients may start at once (it waits for this grid before it
  // reads the tangents)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ LayerP s_lp[kPrepLayers];
  __shared__ LayerD s_ld[kPrepLayers];
  const unsigned I = L - 1;
  const unsigned t0 = blockIdx.x * kPrepThreads, t1 = min(t0 + kPrepThreads, n_items);
  // interfaces, counted over all slownesses; a slowness's layers follow the one's before
  const unsigned q0 = t0 / kPrepItems, q1 = (t1 - 1) / kPrepItems;
  const unsigned e0 = q0 + q0 / I, e1 = q1 + q1 / I + 1;
  for (unsigned e = e0 + threadIdx.x; e <= e1; e += blockDim.x) {
    const unsigned j = e / L;
    const int l = (int)(e - j * L);
    const LayerP lp = layer_terms(tab, L, l, p[j]);
    s_lp[e - e0] = lp;
    s_ld[e - e0] = layer_derivs(tab, L, l, p[j], lp);
  }
  __syncthreads();
  const unsigned t = t0 + threadIdx.x;
  if (t >= t1) return;
  const unsigned q = t / kPrepItems, j = q / I;
  const int item = (int)(t - q * kPrepItems), i = (int)(q - j * I);
  const size_t idx = q, e = (size_t)q + j;
  const int s = (int)(q + j - e0);
  const double pj = p[j];
  const LayerP& up = s_lp[s];
  const LayerP& lo = s_lp[s + 1];
  if (item == 6) {
    lay[e] = up;
    dlay[e] = s_ld[s];
    if (i == L - 2) {
      lay[e + 1] = lo;
      dlay[e + 1] = s_ld[s + 1];
    }
    coef[idx] = interface_coeffs(pj, i, up, lo);
    return;
  }
  cd c[10];
  interface_tangent_col(pj, i, up, s_ld[s], lo, s_ld[s + 1], item, c);
  for (int k = 0; k < 10; ++k) tan[idx].t[k][item] = c[k];
}

static kr_status launch_prep(const double* layers, int L, const double* p, int n_p, LayerP* lay,
                             LayerD* dlay, Iface* coef, ScatTan* tan, cudaStream_t st,
                             const char* what) {
  const long long n_items = (long long)n_p * (L - 1) * kPrepItems;  // 2^31 tangents are 294 GB
  if (n_items > 0x7fffffffLL) return KR_ERR_TOO_LARGE;
  const unsigned n = (unsigned)n_items;
  deriv_prep_kernel<<<(n + kPrepThreads - 1) / kPrepThreads, kPrepThreads, 0, st>>>(
      layers, L, p, n, lay, dlay, coef, tan);
  return check_launch(what);
}

}  // namespace kr
