// Device side of the frequency sums of the adjoint (adjoint_rays in kr_adjoint.cuh): every
// warp adds its 32 lanes' per-step adjoints into its own rows of shared memory (a fixed order:
// deterministic), and the block contracts the summed rows with the coefficient tangents and
// phase-derivative factors once.
#pragma once

#include "kr_adjoint.cuh"
#include "kr_phase.cuh"
#include "kr_sweep.cuh"

namespace kr {

// ------------------------------------------------------------------------------------------
// Phase factors ea, eb of one lane for the derivative sweeps, on tiles of the grid's line
// (kr_phase.cuh): lo[j] = exp(j delta c), j < 16, shared by the block, and, per warp and pass of
// 32 frequencies from kb, hm[m], m < 2: the forward sweep's hi mid at frequency kb + 16 m, so a
// lookup is one product of two reads at fixed offsets.  The derivatives need ea and eb
// themselves in the reverse sweep, so these two are tabulated, not P, Q, S.
//
// hm is exp(omega_{kb + 16 m} c) as the forward sweep rounds it, not the closer direct exp: the
// rounding of omega_{128 u} c is common to a tile's frequencies, and a misfit's adjoint made from
// the forward sweep's R meets this sweep's R in sums over frequency where all but their difference
// cancels.  With direct exps the water layer's alpha and h gradients of 5- to 31-layer models on 4
// to 63 slownesses had errors of up to 1.3e-12 of the largest entry, instead of 3e-14.
//
// Models of up to kRayTabLayers layers tabulate: a 51-layer block of the batched gradient is
// 113 KB (110.4 KB and static arrays), two per SM; from 52 layers the table would cost a resident
// block.  Deeper models that the
// forward sweep tabulates (to kPairLayers) evaluate exponentials with the same rounding of the
// tile's first phase (PhaseLine); beyond, both sides take exp of omega c directly.  Every derivative
// kernel applies the same rules, so they agree bit for bit.
// ------------------------------------------------------------------------------------------
constexpr int kRayTabLayers = 51;
__host__ __device__ inline bool ray_table_model(int n_layers) { return n_layers <= kRayTabLayers; }

struct RayTable {
  const cd* lo;  // the lane's lo entry of phase 0 ([2 (L - 1)][16])
  const cd* hm;  // the lane's hm entry of phase 0 ([2 (L - 1)][2])
  __device__ __forceinline__ cd a(int l) const { return hm[4 * l] * lo[2 * kPhLo * l]; }
  __device__ __forceinline__ cd b(int l) const {
    return hm[4 * l + 2] * lo[2 * kPhLo * l + kPhLo];
  }
  __device__ __forceinline__ bool cheap() const { return true; }
  __device__ __forceinline__ bool grows() const { return false; }  // such warps do without a table
};

__host__ __device__ inline size_t ray_lo_values(int n_layers) {
  return (size_t)kPhLo * 2 * (n_layers - 1);
}
__host__ __device__ inline size_t ray_hm_values(int n_layers) { return 4 * (size_t)(n_layers - 1); }
__host__ __device__ inline size_t ray_table_bytes(int n_layers, int warps) {
  return sizeof(cd) * (ray_lo_values(n_layers) + warps * ray_hm_values(n_layers));
}

// Block-cooperative: the lo entries; returns whether this thread's are usable.  The caller
// synchronises.
__device__ __forceinline__ bool ray_lo_fill(const GridLine& g, int n_layers, const LayerP* lay,
                                            cd* lo) {
  bool ok = true;
  for (int e = threadIdx.x; e < 2 * (n_layers - 1) * kPhLo; e += blockDim.x) {
    const cd v = cexp_(((double)(e % kPhLo) * g.d) * sweep_exponent(lay, e / kPhLo));
    ok &= phase_usable(v);
    lo[e] = v;
  }
  return ok;
}

// exp(a + b) without the rounding of a + b: the sum's remainder (Knuth's two-sum) enters to first
// order, exactly enough as it is below an ulp of the sum.
__device__ __forceinline__ cd cexp_sum(cd a, cd b) {
  const cd s = a + b;
  const double tx = s.x - a.x, ty = s.y - a.y;
  const cd r = mk((a.x - (s.x - tx)) + (b.x - tx), (a.y - (s.y - ty)) + (b.y - ty));
  const cd v = cexp_(s);
  return v + v * r;
}

// Warp-cooperative: the hm entries of the pass from frequency kb; returns (warp-uniform) whether
// all are usable.
__device__ __forceinline__ bool ray_hm_fill(const double2* __restrict__ omega, int n_w, int kb,
                                            int n_layers, const LayerP* lay, cd* hm) {
  bool bad = false;
  const int lane = threadIdx.x & 31;
  // lanes take m = lane & 1 of phase id; past the grid's end the entry is not used
  const GridLine g = grid_line(omega, n_w);
  const double2 w = omega[min(kb & ~(kPhTile - 1), n_w - 1)];
  const cd mid = (double)((kb & (kPhTile - 1)) + kPhLo * (lane & 1)) * g.d;
  for (int e = lane; e < 4 * (n_layers - 1); e += 32) {
    const cd c = sweep_exponent(lay, e >> 1);
    const cd v = cexp_sum(mk(w.x, w.y) * c, mid * c);
    bad |= !phase_usable(v);
    hm[e] = v;
  }
  bad = __any_sync(0xffffffffu, bad);
  __syncwarp();
  return !bad;
}

// The lane's table for a warp whose hm entries are at `hm`.
__device__ __forceinline__ RayTable ray_table(const cd* lo, const cd* hm) {
  const int lane = threadIdx.x & 31;
  return RayTable{lo + (lane & (kPhLo - 1)), hm + (lane >> 4)};
}

// Whether frequency k = w of the grid is on its line.
__device__ __forceinline__ bool on_line(const GridLine& g, int k, double2 w) {
  return fabs(w.x - fma((double)k, g.d.x, g.w0.x)) <= g.tol &&
         fabs(w.y - fma((double)k, g.d.y, g.w0.y)) <= g.tol;
}

// Phases of one frequency by direct exponentials.  On a tile of the grid's line, for a model that
// the forward sweep tabulates, exp(omega_k c) = exp(omega_{128 u} c + (k - 128 u) delta c) with the
// first product rounded as there: without it, gradients of 49- to 66-layer models made from the
// forward's R are off by 2.5e-14 of their largest component, with it by less than 1e-15.  Elsewhere
// w0 is the frequency itself and dw zero.
struct PhaseLine {
  cd w0, dw;
  const LayerP* lay;
  __device__ __forceinline__ cd at(cd c) const {
    // the remainder of the sum for |b| <= |a| (Dekker); otherwise, in the grid's first tile, the
    // rounding it leaves is the frequency's own
    const cd a = w0 * c, b = dw * c, s = a + b, r = b - (s - a);
    const cd v = cexp_(s);
    return cmac(v, v, r);
  }
  __device__ __forceinline__ cd a(int l) const { return at(lay[l].ca); }
  __device__ __forceinline__ cd b(int l) const { return at(lay[l].cb); }
  __device__ __forceinline__ bool cheap() const { return false; }
  __device__ __forceinline__ bool grows() const { return false; }
};
// The same for a warp with growing phases: in the frequency sums a sweep of its own (as a flag of the
// other's, the second way of the step cost deep models 5 to 8 %), in the per-step contraction, with
// few registers to spare, a flag (a third sweep spills: 64 x 1024 Jacobian of 21 layers 108.5 us
// against 106.6).
struct PhaseGrown : PhaseLine {
  __device__ __forceinline__ explicit PhaseGrown(const PhaseLine& p) : PhaseLine(p) {}
  __device__ __forceinline__ bool grows() const { return true; }
};
struct PhaseEither : PhaseLine {
  bool grow;
  __device__ __forceinline__ PhaseEither(const PhaseLine& p, bool g) : PhaseLine(p), grow(g) {}
  __device__ __forceinline__ bool grows() const { return grow; }
};
__device__ __forceinline__ bool ray_line_model(int n_layers) { return n_layers <= kPairLayers; }

// Whether a frequency of the warp has growing phases.  All 32 lanes call it.
__device__ __forceinline__ bool warp_grows(bool valid, cd w) {
  return __any_sync(0xffffffffu, valid && phases_grow(w));
}

// The source of frequency k = w; `on`: its tile is on the line and the forward sweep's phases of it
// come from a table.
__device__ __forceinline__ PhaseLine phase_line(bool on, const double2* __restrict__ omega, int n_w,
                                                int k, cd w, const LayerP* lay) {
  if (!on) return PhaseLine{w, mk(0.0, 0.0), lay};
  const double2 w0 = omega[k & ~(kPhTile - 1)];
  return PhaseLine{mk(w0.x, w0.y), (double)(k & (kPhTile - 1)) * grid_line(omega, n_w).d, lay};
}

// Staging of the warp sums of 12 explicit values per lane (the dual adjoint of the
// Hessian-vector products): a padded 32 x 13 tile.  Tile row stride in complex values:
__host__ __device__ constexpr int stage_stride() { return kSumVals + 1; }

// acc_row[c] += sum over the warp's lanes of v[c], c < 12.  24 lanes (c, g) add the 16 rows of
// row group g in column c, a shuffle combines the two groups; a fixed order (deterministic).
// All 32 lanes call it.
__device__ __forceinline__ void warp_add12(const cd v[kSumVals], cd* stage, cd* acc_row) {
  constexpr int P = kSumVals, S = P + 1;
  const int lane = threadIdx.x & 31;
  cd* mine = stage + lane * S;
#pragma unroll
  for (int k = 0; k < P; ++k) mine[k] = v[k];
  __syncwarp();
  if (lane < 2 * P) {
    const int c = lane % P, g = lane / P;
    cd s = stage[(16 * g) * S + c];
#pragma unroll
    for (int r = 1; r < 16; ++r) s = s + stage[(16 * g + r) * S + c];
    s.x += __shfl_down_sync(0x00ffffffu, s.x, P);
    s.y += __shfl_down_sync(0x00ffffffu, s.y, P);
    if (lane < P) acc_row[c] = acc_row[c] + s;
  }
  __syncwarp();
}

// ------------------------------------------------------------------------------------------
// Sums of the ray sweep (adjoint_rays).  The 12 adjoints of a step are products of two
// components of v = (g1, g2, x1, x2) or of (wz, x), so their sums over a warp's 32
// frequencies are entries of the 8 x 8 real matrix V V^T (V: 8 real components x 32
// frequencies) and of the 4 x 4 blocks Z X^T: FP64 matrix instructions (m8n8k4) form the
// products and the sums together.  On this GPU they run at the vector FMA's rate on the same
// pipe (37.1 TFLOP/s measured against 34-36), so what they save is instructions and shared
// memory: 12 matrix instructions, 6 stores and 16 loads of one double per lane against 56
// FP64 operations, 12 stores, 16 complex loads and 30 adds for explicit products through a
// transposing tile.  With the ray sweep: gradient of 64 slownesses x 1024 frequencies x 21
// layers 110.6 -> 80.7 us, a batch of 96 uneven models 17.8 -> 13.4 ms.
//
// Staging of a warp: rows g1, g2, x1, x2, wz1, wz2 of 32 complex values (lane = frequency),
// padded to 36 so that a half-warp's fragment loads (two rows x 4 frequencies x 2 parts) fall
// on 32 different banks.
//
// A step's sums are a row of 24 doubles; kRow(re / im of entry) below.
// ------------------------------------------------------------------------------------------
constexpr int kRayStride = 36;
constexpr int kRayStage = 6 * kRayStride;  // complex values per warp
constexpr int kRayRow = 24;                // doubles per step and warp

// Bytes of `warps` warps' staging rows, or of the layer terms and roots a block's prologue keeps
// in their place where those are larger (deep models).
__host__ __device__ inline size_t ray_stage_bytes(int L, int warps) {
  const size_t a = sizeof(cd) * kRayStage * (size_t)warps;
  const size_t b = (sizeof(LayerP) + sizeof(LayerRoots)) * (size_t)L;
  return a > b ? a : b;
}

// Shared memory of the ray sums for `warps` warps: per warp L rows and its staging rows.
__host__ __device__ inline size_t raysum_smem_bytes(int L, int warps) {
  return (size_t)warps * (sizeof(double) * kRayRow * sum_rows(L) + sizeof(cd) * kRayStage);
}

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// row[24] += the sums over the warp of the products of one step.  Fragments (m8n8k4): lane
// holds A[lane / 4][lane % 4], B[lane % 4][lane / 4], C[lane / 4][2 (lane % 4) + {0, 1}].
// Entry (a, b) of the complex products sits, after combining the two real rows of a, as Re in
// lane 8 a + b and Im in lane 8 a + 4 + b.
__device__ __forceinline__ void ray_add(const Ray& g, const Ray& x, const Ray& wz, cd* stage,
                                        double* row) {
  const int lane = threadIdx.x & 31;
  cd* mine = stage + lane;
  mine[0 * kRayStride] = g.a;
  mine[1 * kRayStride] = g.b;
  mine[2 * kRayStride] = x.a;
  mine[3 * kRayStride] = x.b;
  mine[4 * kRayStride] = wz.a;
  mine[5 * kRayStride] = wz.b;
  __syncwarp();
  const double* sd = reinterpret_cast<const double*>(stage);
  const int k = lane & 3, r = lane >> 2;
  // V V^T, two accumulators (each a chain of four)
  const double* v = sd + 2 * ((r >> 1) * kRayStride + k) + (r & 1);
  double c0 = 0.0, c1 = 0.0, d0 = 0.0, d1 = 0.0;
#pragma unroll
  for (int m = 0; m < 8; m += 2) {
    const double u0 = v[8 * m], u1 = v[8 * (m + 1)];
    dmma884(c0, c1, u0, u0);
    dmma884(d0, d1, u1, u1);
  }
  // Z X^T: rows / columns 0-3 take the first 4 of 8 frequencies, 4-7 the other 4; the two
  // diagonal blocks of the result are the sums
  const int e = r & 3, f0 = (r >> 2) * 4 + k;
  const double* zx = sd + 2 * ((e >> 1) * kRayStride + f0) + (e & 1);
  double p0 = 0.0, p1 = 0.0;
#pragma unroll
  for (int m = 0; m < 4; ++m)
    dmma884(p0, p1, zx[2 * (4 * kRayStride + 8 * m)], zx[2 * (2 * kRayStride + 8 * m)]);
  c0 += d0;
  c1 += d1;
  // (row 2a: re x {re, im}, row 2a + 1: im x {re, im}) -> Re in the even row, Im in the odd
  const bool odd = (r & 1) != 0;
  const double cp = __shfl_xor_sync(0xffffffffu, c1, 4), pp = __shfl_xor_sync(0xffffffffu, p1, 4);
  double val = odd ? c0 + cp : c0 - cp;
  const double ph = odd ? p0 + pp : p0 - pp;
  // lanes 16, 17, 20, 21 (the redundant entries (x1, g)) take the phase sums z_a x_a of both
  // frequency sets, lanes 8 and 12 (the redundant (g2, g1)) take (x2, x2)
  const int src = (2 * k + (r & 1)) * 4 + k;  // for k < 2: entry (a = k, a) of the first set
  const double q0 = __shfl_sync(0xffffffffu, ph, src & 31);
  const double q1 = __shfl_sync(0xffffffffu, ph, (src + 18) & 31);
  const double x22 = __shfl_sync(0xffffffffu, val, odd ? 31 : 27);
  if ((r >> 1) == 2 && k < 2) val = q0 + q1;
  if ((r >> 1) == 1 && k == 0) val = x22;
  if (lane < kRayRow) row[lane] += val;
  __syncwarp();  // the staging rows are read before the next step's overwrite them
}

// The 12 complex sums of a step (order of ScatTan, then fa, fb) from its row.
__device__ __forceinline__ void ray_row_sums(const double* row, cd out[kSumVals]) {
  auto at = [&](int a, int b) { return mk(row[8 * a + b], row[8 * a + 4 + b]); };
  out[0] = at(0, 0);
  out[1] = 2.0 * at(0, 1);
  out[2] = at(1, 1);
  out[3] = at(2, 2);
  out[4] = 2.0 * at(2, 3);
  out[5] = at(1, 0);
  out[6] = 2.0 * at(0, 2);
  out[7] = 2.0 * at(1, 2);
  out[8] = 2.0 * at(0, 3);
  out[9] = 2.0 * at(1, 3);
  out[10] = 2.0 * at(2, 0);
  out[11] = 2.0 * at(2, 1);
}

// The summing sink of one lane: seed 2 conj(R - R_obs) (misfit) or conj(gR) (cotangent gR).
struct RaySumSink {
  bool valid;
  bool vjp;          // seed with conj(gR) instead of 2 conj(R - R_obs)
  const double2* obs;  // R_obs or gR at this (p, omega)
  double2* R_out;      // R at this (p, omega), or nullptr
  double* acc;         // this warp's sum rows
  cd* stage;           // this warp's staging rows
  int I;
  cd res;
  __device__ cd reflectivity(cd R) {
    res = mk(0.0, 0.0);
    if (!valid) return mk(0.0, 0.0);
    if (R_out) *R_out = make_double2(R.x, R.y);
    const double2 o = *obs;
    if (vjp) return mk(o.x, -o.y);  // conj(gR)
    res = mk(R.x - o.x, R.y - o.y);
    return mk(2.0 * res.x, -2.0 * res.y);  // 2 conj(res)
  }
  __device__ void top(cd f0) {  // row I, first entry (layer 0's phase term)
    if (!valid) f0 = mk(0.0, 0.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      f0.x += __shfl_down_sync(0xffffffffu, f0.x, o);
      f0.y += __shfl_down_sync(0xffffffffu, f0.y, o);
    }
    if ((threadIdx.x & 31) == 0) {
      acc[(size_t)I * kRayRow] += f0.x;
      acc[(size_t)I * kRayRow + 1] += f0.y;
    }
  }
  __device__ void ray(int i, Ray g, Ray x, Ray wz, const S3&, cd, cd) {
    if (!valid) g = x = wz = Ray{mk(0.0, 0.0), mk(0.0, 0.0)};  // a lane without a frequency
    ray_add(g, x, wz, stage, acc + (size_t)i * kRayRow);
  }
};

// Zeroes the warps' sum rows (block-cooperative; the caller synchronises afterwards).
__device__ __forceinline__ void sums_zero(double* acc_all, int L, int warps) {
  const int n = warps * (int)sum_rows(L) * kRayRow;
  for (int k = threadIdx.x; k < n; k += blockDim.x) acc_all[k] = 0.0;
}

// Adds the warps' rows into warp 0's (fixed order), turns each row into its 12 complex sums in
// place (24 doubles either way), then thread l < L contracts layer l into out[k L + l]
// (k = alpha, beta, rho, h).  Contains block barriers; all threads call it.
__device__ __forceinline__ void sums_finish(double* acc_all, int L, int warps,
                                            const ScatTan* __restrict__ tan,
                                            const LayerD* __restrict__ dlay, double* out) {
  const int n = (int)sum_rows(L) * kRayRow, I = L - 1;
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    double s = acc_all[k];
    for (int wi = 1; wi < warps; ++wi) s += acc_all[wi * n + k];
    acc_all[k] = s;
  }
  __syncthreads();
  cd* sums = reinterpret_cast<cd*>(acc_all);
  for (int i = threadIdx.x; i <= I; i += blockDim.x) {
    cd v[kSumVals];
    if (i < I) {
      ray_row_sums(acc_all + (size_t)i * kRayRow, v);
    } else {
#pragma unroll
      for (int k = 0; k < kSumVals; ++k) v[k] = mk(0.0, 0.0);
      v[10] = mk(acc_all[(size_t)I * kRayRow], acc_all[(size_t)I * kRayRow + 1]);
    }
    for (int k = 0; k < kSumVals; ++k) sums[(size_t)i * kSumVals + k] = v[k];
  }
  __syncthreads();
  for (int l = threadIdx.x; l < L; l += blockDim.x) {
    double v[4];
    sums_contract_layer(l, L, sums, tan, dlay, v);
    out[0 * L + l] = v[0];
    out[1 * L + l] = v[1];
    out[2 * L + l] = v[2];
    out[3 * L + l] = v[3];
  }
}

}  // namespace kr
