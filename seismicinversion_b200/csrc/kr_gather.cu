// Discrete-wavenumber gather: Bessel-weighted slowness sum and the omega -> t step.
//
// kr_bessel_sum: one thread per (offset, omega) and slowness slice.  Blocks are
// 32 frequencies x 8 offsets; the slowness range is split into slices (grid.x) so the grid
// fills the 148 SMs several times over; each slice writes its partial U to the workspace and
// a second kernel adds the slices in a fixed order (bit-reproducible).  J0 is evaluated on
// the fly in registers (FP64): Hankel's asymptotic expansion above x = 25 with cos/sin
// carried along the slowness loop by rotation (exact anchors every 32 steps), a piecewise
// Taylor table below; R[p][omega] arrives through shared memory in tiles of 32 slownesses
// x 32 frequencies (cp.async, a ring of three) shared by the block's 8 offsets.
//
// kr_traces: builds the half spectrum conj(U S) (DC and Nyquist zero) and runs a batched
// cuFFT Z2D: for a Hermitian spectrum H, the forward DFT the reference applies
// (np.fft.fft) equals the inverse real transform of conj(H).  The decay exp(-gamma t) is
// applied by a last elementwise kernel.
#include <cufft.h>
#include <stdio.h>

#include <mutex>
#include <vector>

#include "kr_bessel.cuh"
#include "kr_internal.cuh"
#include "kr_j0_table.h"

namespace kr {

constexpr int kBsW = 32;  // frequencies per block
constexpr int kBsR = 8;   // offsets per block

// ---------------------------------------------------------------------------------------
// J0 for large arguments: Hankel's asymptotic expansion (Abramowitz & Stegun 9.2.5,
// 9.2.9-9.2.10) with the coefficients a_k(0) = prod_{j=1..k} (-(2j-1)^2) / (k! 8^k):
//   J0(x) = sqrt(2 / (pi x)) [P(x) cos(x - pi/4) - Q(x) sin(x - pi/4)]
//         = sqrt(1 / (pi x)) [(P + Q) cos x + (P - Q) sin x],
//   P = sum_m (-1)^m a_{2m} x^{-2m},  Q = sum_m (-1)^m a_{2m+1} x^{-2m-1}.
// With 7 terms each the truncation error is below 7e-16 absolute for x >= 25 (checked
// against SciPy's j0); below 25 the kernel uses the Taylor table of kr_j0_table.h.
// ---------------------------------------------------------------------------------------
constexpr double kJ0X0 = 25.0;
constexpr int kJ0Terms = 7;

__host__ __device__ constexpr double hankel_a(int k) {
  double num = 1.0, den = 1.0;
  for (int j = 1; j <= k; ++j) {
    num *= -(double)((2 * j - 1) * (2 * j - 1));
    den *= 8.0 * j;
  }
  return num / den;
}
__host__ __device__ constexpr double hankel_p(int m) { return (m % 2 ? -1.0 : 1.0) * hankel_a(2 * m); }
__host__ __device__ constexpr double hankel_q(int m) { return (m % 2 ? -1.0 : 1.0) * hankel_a(2 * m + 1); }

// The first NT terms of P and x Q at q = 1 / x^2.  The first omitted terms bound the truncation
// error (A&S 9.2.10); the absolute J0 error is below 7e-16 for NT = 7 at x >= 25 and below 1e-16
// for NT = 5 at x >= 60, NT = 4 at x >= 100, NT = 3 at x >= 300 and NT = 2 at x >= 3000.
template <int NT>
__device__ __forceinline__ void hankel_series(double q, double& P, double& Q) {
  P = hankel_p(NT - 1);
  Q = hankel_q(NT - 1);
#pragma unroll
  for (int m = NT - 2; m >= 0; --m) {
    P = fma(P, q, hankel_p(m));
    Q = fma(Q, q, hankel_q(m));
  }
}

// J0(x) for x >= kJ0X0 given c = cos x, s = sin x.
__device__ __forceinline__ double j0_asymptotic(double x, double c, double s) {
  const double amp = rsqrt(3.14159265358979323846 * x);  // sqrt(1 / (pi x))
  const double y = 3.14159265358979323846 * (amp * amp);  // 1 / x
  const double q = y * y;
  double P = hankel_p(kJ0Terms - 1), Q = hankel_q(kJ0Terms - 1);
#pragma unroll
  for (int m = kJ0Terms - 2; m >= 0; --m) {
    P = fma(P, q, hankel_p(m));
    Q = fma(Q, q, hankel_q(m));
  }
  Q *= y;
  return amp * fma(P + Q, c, (P - Q) * s);
}

// J0(x) for 0 <= x < 25 from the piecewise Taylor table (kr_j0_table.h, staged in shared
// memory with rows padded to kJ0Row doubles so that lanes on different intervals fall on
// different banks): interval and offset t by j0_interval, degree-15 Horner in t.
// Absolute error below 5e-16 against SciPy's j0 on [0, 25).
constexpr int kJ0Row = kJ0TabDegree + 2;
__device__ __forceinline__ double j0_table(const double* s_j0, double x) {
  double t;
  const double* a = s_j0 + j0_interval(x, kJ0TabIntervals, t) * kJ0Row;
  double v = a[kJ0TabDegree];
#pragma unroll
  for (int n = kJ0TabDegree - 1; n >= 0; --n) v = fma(v, t, a[n]);
  return v;
}

// Slowness steps between exact sincos anchors when p is an arithmetic progression.
constexpr int kRotSteps = 32;
// R rows are staged through shared memory in tiles of kSub slownesses x 32 frequencies
// (16 KB) in a ring of three with cp.async: the 8 offset warps of a block read each R
// element from shared memory instead of each loading it from L1 / L2, two tiles are in
// flight while one is summed, and one block barrier per tile suffices (the barrier that
// publishes tile t also shows every warp done with tile t - 1, whose buffer then takes
// tile t + 2).  kSub equals the rotation anchor spacing.  One warp in turn forms the next tile's
// factors of the slowness alone.
constexpr int kSub = kRotSteps;
constexpr int kRing = 3;
constexpr size_t kRingBytes = sizeof(double2) * kRing * kSub * kBsW;  // dynamic shared memory

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem),
               "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;\n" ::); }

// Block-cooperative: R rows [j0, j0 + ns) x frequencies [iw0, iw0 + 32) into `tile`,
// zero-filled (no global read) outside the grid.  Warp ty copies rows ty, ty + 8, ...;
// lane copies frequency iw0 + lane (one coalesced 512-byte row per warp and copy).
__device__ __forceinline__ void stage_R(double2 (*tile)[kBsW], const double2* __restrict__ R,
                                        int j0, int ns, int iw0, int n_w) {
  const int ty = threadIdx.y, lane = threadIdx.x;
  const bool col_ok = iw0 + lane < n_w;
  const double2* src = R + (size_t)(j0 + ty) * n_w + iw0 + lane;
  const size_t stride = (size_t)kBsR * n_w;
#pragma unroll
  for (int i = 0; i < kSub / kBsR; ++i) {
    const int row = ty + i * kBsR;
    const bool ok = col_ok && row < ns;
    cp_async16(&tile[row][lane], ok ? src + i * stride : R, ok ? 16 : 0);
  }
}

// Terms of one staged tile for one thread on the fast path.  With z = 1 / (omega r),
//   sqrt(pi omega r) f_j J0(x_j) = (f_j / sqrt p_j) P u + (f_j / p_j^1.5) Q v,
//   u = cos x + sin x, v = (cos x - sin x) z, P and Q at 1 / x^2 = z^2 / p_j^2:
// what depends on the slowness alone is staged, what depends on the thread alone waits until
// the end, 2 NT + 5 operations a term with the two of the sum (2 NT + 6 with 1 / x formed per
// term and the weight applied to J0).  The tile starts from an exact cos and sin; from one
// slowness to the next (u, v) turn by the step's angle d: in three shears (3 operations; tn =
// tan(d / 2) / z, sn = z sin d), or, where a lane's d lies near half a turn and tan(d / 2) is
// large, by products (4 operations; cs = cos d, s1 = sin d / z, sn).
struct TileTurn {
  double tn, sn, cs, s1;
};

template <int NT, bool SHEAR, int M>
__device__ __forceinline__ void fast_terms(const double2* __restrict__ w_p,
                                           const double* __restrict__ q_p,
                                           const double2* __restrict__ r_p, int m, double z2,
                                           const TileTurn& d, double u, double v, double& ax,
                                           double& ay) {
#pragma unroll 8
  for (int k = 0; k < (M > 0 ? M : m); ++k) {
    const double2 w = w_p[k];
    const double2 rv = r_p[k * kBsW];
    double P, Q;
    hankel_series<NT>(q_p[k] * z2, P, Q);
    const double t = fma(w.x, P * u, w.y * (Q * v));
    if (SHEAR) {
      u = fma(d.tn, v, u);
      v = fma(-d.sn, u, v);
      u = fma(d.tn, v, u);
    } else {
      const double u2 = fma(u, d.cs, v * d.s1);
      v = fma(v, d.cs, -u * d.sn);
      u = u2;
    }
    ax = fma(t, rv.x, ax);
    ay = fma(t, rv.y, ay);
  }
}

template <int NT>
__device__ __forceinline__ void fast_tile(const double2* w_p, const double* q_p,
                                          const double2* r_p, int m, bool shear, double z2,
                                          const TileTurn& d, double u, double v, double& ax,
                                          double& ay) {
  // full tiles run a loop of compile-time length (no remainder handling)
  if (m == kSub && shear)
    fast_terms<NT, true, kSub>(w_p, q_p, r_p, kSub, z2, d, u, v, ax, ay);
  else if (m == kSub)
    fast_terms<NT, false, kSub>(w_p, q_p, r_p, kSub, z2, d, u, v, ax, ay);
  else
    fast_terms<NT, false, 0>(w_p, q_p, r_p, m, z2, d, u, v, ax, ay);
}

// One thread per (omega, offset) and slowness slice.  Grid: x = slowness slice, y = offset
// group, z = frequency tile, so the hardware starts the low-frequency tiles (small J0
// arguments, the slowest blocks) first and the cheap high-frequency tiles fill the tail.
// Per tile the block stages the slownesses' factors in shared memory with a check whether the
// tile continues the slice's arithmetic progression (to 4.5 ulp); inside such a tile cos / sin of
// x_j = (omega p_j) r advance by one rotation per slowness from an exact anchor.  A tile whose
// arguments stay below 25 sums from the table alone, one that crosses 25 decides term by term.
// omega is factored out of the weight: U = omega * sum_j J0(x_j) (pw_j dp) R_j.  Four blocks of 256
// threads per SM (64 registers): with three distinct operands in most of its instructions the
// kernel is bound by the register ports and by each warp's dependency chains, so more resident
// warps help despite some spills.  Two offsets per thread share the loads of R and of factors
// already multiplied by the weight (11 operations a term instead of 14), but leave 24 or 16 warps
// per SM: 2.58 to 2.9 ms on 8192 slownesses x 2047 frequencies x 100 offsets against 2.47 ms,
// which took 2.59 with 16 operations a term, chunks of 128 slownesses between drained rings, and
// per-term branches below 25 (2048 x 511 x 37: 127 -> 100 us, 1000 x 300 x 100: 118 -> 89).
__global__ void __launch_bounds__(kBsW * kBsR, 4)
bessel_partial_kernel(const double2* __restrict__ R, const double* __restrict__ p,
                      const double* __restrict__ pw, int n_p, double dp,
                      const double* __restrict__ omega, int n_w,
                      const double* __restrict__ offsets, int n_r, int p_per_slice,
                      double2* __restrict__ partial) {
  __shared__ double2 s_pf[2][kSub];  // (p_j, f_j) with f_j = pw_j dp
  __shared__ double2 s_w[2][kSub];   // (f_j / sqrt p_j, f_j / p_j^1.5)
  __shared__ double s_q[2][kSub];    // 1 / p_j^2
  __shared__ int s_line[2];          // the tile lies on the progression
  __shared__ double s_j0[kJ0TabIntervals * kJ0Row];
  extern __shared__ __align__(16) unsigned char s_dyn[];
  double2(*s_R)[kSub][kBsW] = reinterpret_cast<double2(*)[kSub][kBsW]>(s_dyn);  // [kRing]
  const int tid = threadIdx.y * kBsW + threadIdx.x;
  for (int e = tid; e < kJ0TabIntervals * kJ0Row; e += kBsW * kBsR) {
    const int k = e / kJ0Row, n = e - k * kJ0Row;
    s_j0[e] = n <= kJ0TabDegree ? kJ0Taylor[k][n] : 0.0;  // made visible by the first barrier
  }
  const int lane = threadIdx.x;
  const int iw0 = blockIdx.z * kBsW;
  const int ir = blockIdx.y * kBsR + threadIdx.y;
  const int j_begin = blockIdx.x * p_per_slice;
  const int j_end = min(n_p, j_begin + p_per_slice);
  const bool working = ir < n_r;  // a warp without an offset only stages
  // lanes beyond the grid repeat its last frequency, so that they take their warp's path
  const double om = omega[min(iw0 + lane, n_w - 1)];
  const double r = working ? offsets[ir] : 0.0;
  const double omr = om * r;
  // z^2 and what it meets stay finite, or x is 0 throughout; for the whole warp, whose lanes
  // vote below
  const bool regular =
      __all_sync(0xffffffffu, (omr >= 1e-100 && omr <= 1e100) || omr == 0.0);
  const double z = omr > 0.0 ? 1.0 / omr : 0.0;
  // Linear model of the slice's slownesses: p_j ~ p0 + (j - j_begin) * step.
  const double p0 = __ldg(p + j_begin);
  const double step =
      (j_end - j_begin >= 2) ? (__ldg(p + j_end - 1) - p0) / (double)(j_end - 1 - j_begin) : 0.0;
  double sd, cdl;
  sincos(omr * step, &sd, &cdl);
  // shears up to 2 pi / 3, where tan(d / 2) is 1.7 (the whole warp, or products)
  const bool shear = __all_sync(0xffffffffu, cdl >= -0.5);
  const double half_tan = sd / (1.0 + cdl);
  double ax = 0.0, ay = 0.0;  // fast-path terms, without the factor 1 / sqrt(pi omega r)
  double bx = 0.0, by = 0.0;  // other terms, complete
  const int n = j_end - j_begin, ntile = (n + kSub - 1) / kSub;
  auto prepare = [&](int t) {  // one warp
    const int b = t & 1, j = t * kSub + lane;
    bool ok = true;
    if (j < n) {
      const double pj = __ldg(p + j_begin + j);
      const double f = __ldg(pw + j_begin + j) * dp;
      const double y = 1.0 / pj;
      const double w = f * rsqrt(pj);
      s_pf[b][lane] = make_double2(pj, f);
      s_w[b][lane] = make_double2(w, w * y);
      s_q[b][lane] = y * y;
      ok = fabs(pj - fma((double)j, step, p0)) <= 1e-15 * fabs(pj);
    }
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) s_line[b] = ok;
  };
  // tiles 0 and 1 now, tile t + 2 in iteration t; every thread commits one group per step (empty
  // ones included), so wait_group 1 at iteration t means tile t has landed
  stage_R(s_R[0], R, j_begin, min(kSub, n), iw0, n_w);
  cp_async_commit();
  if (ntile > 1) stage_R(s_R[1], R, j_begin + kSub, min(kSub, n - kSub), iw0, n_w);
  cp_async_commit();
  if (threadIdx.y == 0) prepare(0);
  for (int t = 0, ring = 0; t < ntile; ++t, ring = ring == kRing - 1 ? 0 : ring + 1) {
    cp_async_wait_1();  // this thread's copies of tile t have landed
    __syncthreads();    // ... and every thread's; every thread is done with tile t - 1
    if (t + 2 < ntile)
      stage_R(s_R[ring == 0 ? kRing - 1 : ring - 1], R, j_begin + (t + 2) * kSub,
              min(kSub, n - (t + 2) * kSub), iw0, n_w);
    cp_async_commit();
    if (t + 1 < ntile && threadIdx.y == (t + 1) % kBsR) prepare(t + 1);
    if (!working) continue;
    const double2* r_p = &s_R[ring][0][lane];
    const double2 *pf_p = s_pf[t & 1], *w_p = s_w[t & 1];
    const double* q_p = s_q[t & 1];
    const int m = min(kSub, n - t * kSub);
    // A falling tile is a rising one from its other end, where its first (least) argument is then.
    const double p_first = pf_p[step > 0.0 ? 0 : m - 1].x, x_first = (om * p_first) * r;
    const bool steady = rising_tile(s_line[t & 1] != 0, fabs(step), p_first, regular);
    // Fast tile: slownesses in arithmetic progression with x >= 25 in every lane, so every term
    // takes the asymptotic branch with the anchor / rotation scheme (no data-dependent branches
    // in the inner loop).  The number of expansion terms follows from the warp's smallest
    // argument.
    const int nt = x_first >= 3000.0 ? 2 : x_first >= 300.0 ? 3 : x_first >= 100.0 ? 4
                 : x_first >= 60.0 ? 5 : x_first >= kJ0X0 ? 7 : 8;
    const int terms = __reduce_max_sync(0xffffffffu, steady ? nt : 8);
    if (terms < 8) {
      double s, c;
      sincos((om * pf_p[0].x) * r, &s, &c);
      const TileTurn d = {half_tan * omr, sd * z, cdl, sd * omr};
      const double u = c + s, v = (c - s) * z, z2 = z * z;
      switch (terms) {
        case 2: fast_tile<2>(w_p, q_p, r_p, m, shear, z2, d, u, v, ax, ay); break;
        case 3: fast_tile<3>(w_p, q_p, r_p, m, shear, z2, d, u, v, ax, ay); break;
        case 4: fast_tile<4>(w_p, q_p, r_p, m, shear, z2, d, u, v, ax, ay); break;
        case 5: fast_tile<5>(w_p, q_p, r_p, m, shear, z2, d, u, v, ax, ay); break;
        default: fast_tile<7>(w_p, q_p, r_p, m, shear, z2, d, u, v, ax, ay); break;
      }
      continue;
    }
    if (steady && __all_sync(0xffffffffu, (om * pf_p[step > 0.0 ? m - 1 : 0].x) * r < kJ0X0)) {
      // every term from the table
#pragma unroll 2
      for (int k = 0; k < m; ++k) {
        const double2 pf = pf_p[k];
        const double2 rv = r_p[k * kBsW];
        const double t = j0_table(s_j0, (om * pf.x) * r) * pf.y;
        bx = fma(t, rv.x, bx);
        by = fma(t, rv.y, by);
      }
    } else if (steady) {
      // the tile crosses x = 25
      double s, c;
      sincos((om * pf_p[0].x) * r, &s, &c);
      const double sn = sd * z, s1 = sd * omr, z2 = z * z;
      double u = c + s, v = (c - s) * z;
#pragma unroll 1
      for (int k = 0; k < m; ++k) {
        const double2 pf = pf_p[k];
        const double2 rv = r_p[k * kBsW];
        const double x = (om * pf.x) * r;
        if (x < kJ0X0) {
          const double t = j0_table(s_j0, x) * pf.y;
          bx = fma(t, rv.x, bx);
          by = fma(t, rv.y, by);
        } else {
          const double2 w = w_p[k];
          double P, Q;
          hankel_series<kJ0Terms>(q_p[k] * z2, P, Q);
          const double t = fma(w.x, P * u, w.y * (Q * v));
          ax = fma(t, rv.x, ax);
          ay = fma(t, rv.y, ay);
        }
        const double u2 = fma(u, cdl, v * s1);
        v = fma(v, cdl, -u * sn);
        u = u2;
      }
    } else {
      // slownesses off the progression or below zero, a negative or extreme omega r: each term by
      // itself (a rotation here for falling tiles costs the others registers: 6000 x 1000 x 10 173 us
      // against 167)
#pragma unroll 1
      for (int k = 0; k < m; ++k) {
        const double2 pf = pf_p[k];
        const double2 rv = r_p[k * kBsW];
        const double x = (om * pf.x) * r;
        double jv;
        if (x < kJ0X0) {
          jv = x > -kJ0X0 ? j0_table(s_j0, fabs(x)) : j0(x);
        } else {
          double s, c;
          sincos(x, &s, &c);
          jv = j0_asymptotic(x, c, s);
        }
        const double t = jv * pf.y;
        bx = fma(t, rv.x, bx);
        by = fma(t, rv.y, by);
      }
    }
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (working && iw0 + lane < n_w) {
    const double amp = omr > 0.0 ? rsqrt(3.14159265358979323846 * omr) : 0.0;
    partial[((size_t)blockIdx.x * n_r + ir) * n_w + iw0 + lane] =
        make_double2(fma(ax, amp, bx) * om, fma(ay, amp, by) * om);
  }
}

// U = sum of the slices' partials: 32 elements per block, eight threads per element (slices s,
// s + 8, ...), whose sums are added in order.
__global__ void __launch_bounds__(256)
reduce_slices_kernel(const double2* __restrict__ partial, int n_slices, size_t n_elem,
                     double2* __restrict__ U) {
  __shared__ double2 s_sum[8][32];
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
  const size_t i = blockIdx.x * (size_t)32 + lane;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  double x = 0.0, y = 0.0;
  if (i < n_elem) {
#pragma unroll 4
    for (int s = part; s < n_slices; s += 8) {
      const double2 v = partial[(size_t)s * n_elem + i];
      x += v.x;
      y += v.y;
    }
  }
  s_sum[part][lane] = make_double2(x, y);
  __syncthreads();
  if (part != 0 || i >= n_elem) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    x += s_sum[k][lane].x;
    y += s_sum[k][lane].y;
  }
  U[i] = make_double2(x, y);
}

// The sum of the slices starts its launch while the last of them finish.
static kr_status launch_reduce(const double2* partial, int n_slices, size_t n_elem, double* U,
                               cudaStream_t st, const char* where) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((n_elem + 31) / 32));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, reduce_slices_kernel, partial, n_slices, n_elem,
                                           reinterpret_cast<double2*>(U));
  if (e != cudaSuccess) set_last_error(where, e);
  return cuda_status(e);
}

// The R ring lives in dynamic shared memory above the 48 KB default (with the static arrays
// ~54 KB per block, four blocks per SM); the limit is raised once per device.
static SmemLimit g_ring_limit;
static kr_status bessel_ring_attribute(const char* where) {
  return raise_smem_limit((const void*)bessel_partial_kernel, kRingBytes, g_ring_limit, where);
}

struct BesselPlan {
  int n_slices;
  int p_per_slice;
  size_t partial_bytes;
};

static int whole_tiles(int n) {
  return n > 0x7fffffff - kSub ? n : (n + kSub - 1) / kSub * kSub;
}

static BesselPlan bessel_plan(int n_p, int n_w, int n_r) {
  BesselPlan b;
  const long long tiles = (long long)((n_w + kBsW - 1) / kBsW) * ((n_r + kBsR - 1) / kBsR);
  // About 96 blocks of 256 threads per SM in total (~24 waves at 4 resident blocks per SM: shorter
  // blocks even out the slow low-frequency tiles; 8192 slownesses x 2047 frequencies x 100 offsets
  // take 2.467 ms, 2.474 at 64 and 2.468 at 160), but no slice shorter than two tiles
  // (2048 x 511 x 37: 100 us, 105 with three tiles, 109 with four; one tile takes 100 there but 175
  // against 163 at 6000 x 1000 x 10, where the slices' prologues weigh more).
  const long long target = 148LL * 96;
  long long s = (target + tiles - 1) / (tiles > 0 ? tiles : 1);
  long long smax = (n_p + 63) / 64;
  if (s > smax) s = smax;
  if (s < 1) s = 1;
  if (s > 65535) s = 65535;
  b.p_per_slice = whole_tiles((int)((n_p + s - 1) / s));
  b.n_slices = (int)((n_p + b.p_per_slice - 1) / b.p_per_slice);
  if (b.n_slices < 1) b.n_slices = 1;
  b.partial_bytes = (size_t)b.n_slices * n_r * n_w * sizeof(double2);
  return b;
}

// ---------------------------------------------------------------------------------------
// Traces
// ---------------------------------------------------------------------------------------
__global__ void half_spectrum_kernel(const double2* __restrict__ U, const double2* __restrict__ S,
                                     int n_r, int nw, double2* __restrict__ X) {
  const int nh = nw + 1;
  const size_t n = (size_t)n_r * nh;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / nh);
    const int k = (int)(i % nh);
    double2 v = make_double2(0.0, 0.0);
    if (k >= 1 && k <= nw - 1) {
      double2 u = U[(size_t)r * (nw - 1) + (k - 1)];
      if (S) {
        double2 s = S[k - 1];
        cd y = mk(u.x, u.y) * mk(s.x, s.y);
        u = make_double2(y.x, y.y);
      }
      v = make_double2(u.x, -u.y);
    }
    X[i] = v;
  }
}

__global__ void decay_kernel(double* __restrict__ tr, const double* __restrict__ decay, int n_r,
                             int nt) {
  const size_t n = (size_t)n_r * nt;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    tr[i] *= decay[i % nt];
}

struct FftEntry {
  int device;
  int nt;
  int batch;
  cufftHandle plan;
  size_t work;
};

static std::mutex g_fft_mu;
static std::vector<FftEntry> g_fft;

// Returns a cached C2R plan (auto work-area allocation off) for nt-point transforms.
static kr_status get_fft_plan(int nt, int batch, FftEntry** out) {
  int dev = 0;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess) {
    set_last_error("kr_traces: cudaGetDevice", ce);
    return KR_ERR_CUDA;
  }
  for (auto& e : g_fft)
    if (e.device == dev && e.nt == nt && e.batch == batch) {
      *out = &e;
      return KR_OK;
    }
  FftEntry e;
  e.device = dev;
  e.nt = nt;
  e.batch = batch;
  if (cufftCreate(&e.plan) != CUFFT_SUCCESS) return KR_ERR_CUFFT;
  if (cufftSetAutoAllocation(e.plan, 0) != CUFFT_SUCCESS) {
    cufftDestroy(e.plan);
    return KR_ERR_CUFFT;
  }
  int n = nt;
  if (cufftMakePlanMany(e.plan, 1, &n, nullptr, 1, nt / 2 + 1, nullptr, 1, nt, CUFFT_Z2D, batch,
                        &e.work) != CUFFT_SUCCESS) {
    cufftDestroy(e.plan);
    set_last_error_msg("kr_traces: cufftMakePlanMany failed");
    return KR_ERR_CUFFT;
  }
  g_fft.push_back(e);
  *out = &g_fft.back();
  return KR_OK;
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace kr

using namespace kr;

extern "C" size_t kr_bessel_sum_workspace_bytes(int32_t n_p, int32_t n_w, int32_t n_r) {
  if (n_p <= 0 || n_w <= 0 || n_r <= 0) return 0;
  return bessel_plan(n_p, n_w, n_r).partial_bytes;
}

extern "C" kr_status kr_bessel_sum(const double* R, const double* p, const double* pw,
                                   int32_t n_p, double dp, const double* omega, int32_t n_w,
                                   const double* offsets, int32_t n_r, double* U,
                                   void* workspace, size_t workspace_bytes, void* stream) {
  if (n_p < 0 || n_w < 0 || n_r < 0) return KR_ERR_INVALID_ARGUMENT;
  if (n_w == 0 || n_r == 0) return KR_OK;
  if (!U || !omega || !offsets) return KR_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  if (n_p == 0) {
    cudaError_t e = cudaMemsetAsync(U, 0, (size_t)n_r * n_w * sizeof(double2), st);
    if (e != cudaSuccess) set_last_error("kr_bessel_sum: memset", e);
    return cuda_status(e);
  }
  if (!R || !p || !pw) return KR_ERR_INVALID_ARGUMENT;
  if (!aligned16(R) || !aligned16(U)) return KR_ERR_INVALID_ARGUMENT;
  if ((n_r + kBsR - 1) / kBsR > 65535 || (n_w + kBsW - 1) / kBsW > 65535)
    return KR_ERR_TOO_LARGE;
  BesselPlan b = bessel_plan(n_p, n_w, n_r);
  if (!workspace || workspace_bytes < b.partial_bytes) return KR_ERR_WORKSPACE;
  double2* partial = reinterpret_cast<double2*>(workspace);
  dim3 grid(b.n_slices, (n_r + kBsR - 1) / kBsR, (n_w + kBsW - 1) / kBsW);
  kr_status a = bessel_ring_attribute("kr_bessel_sum");
  if (a != KR_OK) return a;
  bessel_partial_kernel<<<grid, dim3(kBsW, kBsR), kRingBytes, st>>>(
      reinterpret_cast<const double2*>(R), p, pw, n_p, dp, omega, n_w, offsets, n_r,
      b.p_per_slice, partial);
  kr_status s = check_launch("kr_bessel_sum: partial");
  if (s != KR_OK) return s;
  return launch_reduce(partial, b.n_slices, (size_t)n_r * n_w, U, st, "kr_bessel_sum: reduce");
}

extern "C" size_t kr_traces_workspace_bytes(int32_t n_r, int32_t nw) {
  if (n_r <= 0 || nw <= 1) return 0;
  std::lock_guard<std::mutex> lk(g_fft_mu);
  FftEntry* e = nullptr;
  if (get_fft_plan(2 * nw, n_r, &e) != KR_OK) return 0;
  return align256((size_t)n_r * (nw + 1) * sizeof(double2)) + e->work;
}

extern "C" kr_status kr_traces(const double* U, const double* S, int32_t n_r, int32_t nw,
                               const double* decay, double* traces, void* workspace,
                               size_t workspace_bytes, void* stream) {
  if (n_r < 0 || nw < 0) return KR_ERR_INVALID_ARGUMENT;
  if (n_r == 0) return KR_OK;
  if (nw < 2) return KR_ERR_INVALID_ARGUMENT;
  if (!U || !traces) return KR_ERR_INVALID_ARGUMENT;
  if (!aligned16(U) || (S && !aligned16(S))) return KR_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  std::lock_guard<std::mutex> lk(g_fft_mu);
  FftEntry* e = nullptr;
  kr_status s = get_fft_plan(2 * nw, n_r, &e);
  if (s != KR_OK) return s;
  const size_t xbytes = align256((size_t)n_r * (nw + 1) * sizeof(double2));
  if (!workspace || workspace_bytes < xbytes + e->work) return KR_ERR_WORKSPACE;
  double2* X = reinterpret_cast<double2*>(workspace);
  void* work = static_cast<unsigned char*>(workspace) + xbytes;
  const size_t nx = (size_t)n_r * (nw + 1);
  int blocks = (int)((nx + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  half_spectrum_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<const double2*>(U),
                                               reinterpret_cast<const double2*>(S), n_r, nw, X);
  s = check_launch("kr_traces: half spectrum");
  if (s != KR_OK) return s;
  if (cufftSetStream(e->plan, st) != CUFFT_SUCCESS) return KR_ERR_CUFFT;
  if (e->work && cufftSetWorkArea(e->plan, work) != CUFFT_SUCCESS) return KR_ERR_CUFFT;
  if (cufftExecZ2D(e->plan, reinterpret_cast<cufftDoubleComplex*>(X), traces) != CUFFT_SUCCESS) {
    set_last_error_msg("kr_traces: cufftExecZ2D failed");
    return KR_ERR_CUFFT;
  }
  if (decay) {
    const size_t nt_all = (size_t)n_r * 2 * nw;
    int b2 = (int)((nt_all + 255) / 256);
    if (b2 > 148 * 16) b2 = 148 * 16;
    decay_kernel<<<b2, 256, 0, st>>>(traces, decay, n_r, 2 * nw);
    return check_launch("kr_traces: decay");
  }
  return KR_OK;
}

// ---------------------------------------------------------------------------------------
// Allocation-free variant of kr_bessel_sum.
//
// Some callers cannot allocate device memory at all: a host application that reserved the
// whole GPU in its own pool at start-up and hands out only pointers, a processing system
// that reaches this library through a C/Fortran FFI with device buffers owned by another
// component, or a loop that must not hit cudaMalloc's implicit device synchronisation.
// They pass inputs and the output only; the slice partials live in this file-scope device
// array instead of a caller workspace.  Every GPU that loads the library holds the array
// (16 MiB) until the process exits.
// ---------------------------------------------------------------------------------------
namespace kr {

constexpr size_t kNoAllocScratchBytes = (size_t)16 << 20;
static __device__ __align__(256) unsigned char g_bessel_scratch[kNoAllocScratchBytes];

static std::mutex g_scratch_mu;
struct ScratchSlot {
  void* ctx;   // the context the address belongs to
  void* addr;  // device address of g_bessel_scratch in that context
};
static ScratchSlot g_scratch[kMaxDevices];

// cuCtxGetCurrent through the runtime's driver entry-point table (no link against libcuda).
typedef int (*CtxGetCurrentFn)(void**);
static CtxGetCurrentFn ctx_get_current() {
  static CtxGetCurrentFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<CtxGetCurrentFn>(f);
  }
  return fn;
}

// Device address of g_bessel_scratch in the current device's current context.  The
// host-side symbol is only a stand-in, so the address is looked up (with that device
// current) on the first call per device and again whenever the device's context has changed
// since (cudaDeviceReset makes a new primary context, in which the array lives elsewhere).
static kr_status scratch_address(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_last_error("kr_bessel_sum_noalloc: cudaGetDevice", e);
    return KR_ERR_CUDA;
  }
  if (dev < 0 || dev >= kMaxDevices) {
    set_last_error_msg("kr_bessel_sum_noalloc: device index beyond 63");
    return KR_ERR_TOO_LARGE;
  }
  void* ctx = nullptr;
  CtxGetCurrentFn get = ctx_get_current();
  if (get) get(&ctx);
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  ScratchSlot& slot = g_scratch[dev];
  if (!slot.addr || !ctx || slot.ctx != ctx) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_bessel_scratch);
    if (e != cudaSuccess || !ptr) {
      set_last_error("kr_bessel_sum_noalloc: cudaGetSymbolAddress", e);
      return KR_ERR_CUDA;
    }
    if (!ctx && get) get(&ctx);  // the lookup made the primary context current
    slot.addr = ptr;
    slot.ctx = ctx;
  }
  *out = slot.addr;
  return KR_OK;
}

}  // namespace kr

extern "C" size_t kr_bessel_sum_noalloc_scratch_bytes(void) { return kNoAllocScratchBytes; }

extern "C" kr_status kr_bessel_sum_noalloc(const double* R, const double* p, const double* pw,
                                           int32_t n_p, double dp, const double* omega,
                                           int32_t n_w, const double* offsets, int32_t n_r,
                                           double* U, void* stream) {
  if (n_p < 0 || n_w < 0 || n_r < 0) return KR_ERR_INVALID_ARGUMENT;
  if (n_w == 0 || n_r == 0) return KR_OK;
  if (!U || !omega || !offsets) return KR_ERR_INVALID_ARGUMENT;
  const size_t slice_bytes = (size_t)n_r * n_w * sizeof(double2);
  if (slice_bytes > kNoAllocScratchBytes) {
    char buf[200];
    snprintf(buf, sizeof buf,
             "kr_bessel_sum_noalloc: n_r * n_w = %lld exceeds the static scratch "
             "(16 MiB holds n_r * n_w <= %lld)",
             (long long)n_r * n_w, (long long)(kNoAllocScratchBytes / sizeof(double2)));
    set_last_error_msg(buf);
    return KR_ERR_TOO_LARGE;
  }
  if ((n_r + kBsR - 1) / kBsR > 65535 || (n_w + kBsW - 1) / kBsW > 65535)
    return KR_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  if (n_p == 0) {
    cudaError_t e = cudaMemsetAsync(U, 0, (size_t)n_r * n_w * sizeof(double2), st);
    if (e != cudaSuccess) set_last_error("kr_bessel_sum_noalloc: memset", e);
    return cuda_status(e);
  }
  if (!R || !p || !pw) return KR_ERR_INVALID_ARGUMENT;
  if (!aligned16(R) || !aligned16(U)) return KR_ERR_INVALID_ARGUMENT;
  void* scratch = nullptr;
  kr_status s = scratch_address(&scratch);
  if (s != KR_OK) return s;
  // As many slowness slices as the occupancy target asks for and the scratch holds.  Each
  // slice element is written by exactly one thread before the reduction reads it, so the
  // array needs no clearing between calls.
  BesselPlan b = bessel_plan(n_p, n_w, n_r);
  const int cap = (int)(kNoAllocScratchBytes / slice_bytes);
  int n_slices = b.n_slices < cap ? b.n_slices : cap;
  const int p_per_slice = whole_tiles((n_p + n_slices - 1) / n_slices);
  n_slices = (n_p + p_per_slice - 1) / p_per_slice;
  double2* partial = reinterpret_cast<double2*>(scratch);
  dim3 grid(n_slices, (n_r + kBsR - 1) / kBsR, (n_w + kBsW - 1) / kBsW);
  s = bessel_ring_attribute("kr_bessel_sum_noalloc");
  if (s != KR_OK) return s;
  bessel_partial_kernel<<<grid, dim3(kBsW, kBsR), kRingBytes, st>>>(
      reinterpret_cast<const double2*>(R), p, pw, n_p, dp, omega, n_w, offsets, n_r,
      p_per_slice, partial);
  s = check_launch("kr_bessel_sum_noalloc: partial");
  if (s != KR_OK) return s;
  return launch_reduce(partial, n_slices, (size_t)n_r * n_w, U, st,
                       "kr_bessel_sum_noalloc: reduce");
}
