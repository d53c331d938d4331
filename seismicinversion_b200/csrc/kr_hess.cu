// Exact Hessian of the misfit over every sub-ocean layer's (alpha, beta, rho, h), by pairs of
// layers (kr_hess.cuh), where kr_misfit_hvp runs one dual adjoint per direction.
//
// Kernels (stream-ordered, no host synchronisation):
//   deriv_prep_kernel    : per (p, interface): layer terms, coefficients, tangents
//   hess_rays_kernel     : per (p, omega): forward sweep and ray sweep; leaves X, the phases, g and
//                          K of every step and the seed in the workspace, and the frequency sums
//                          of the adjoints
//   hess_pairs_kernel    : per (p, 16 omega): every pair of layers, summed over its frequencies
//   hess_curvature_kernel: per (p, interface): the adjoint sums times the coefficients' and
//                          phases' second derivatives
//   hess_assemble_kernel : adds blocks and slownesses in a fixed order, writes H
// The first two of slownesses whose steps exceed kStepBytes run in turns.
// Replaces torch.func.hessian of the reference's tau-p misfit (taup_inversion.py:177,
// kennett_torch.py:644-684).
//
// 64 slownesses x 1024 frequencies x 21 layers (79 parameters): 20.1 ms by directions, here
// 0.10 ms for the rays, 0.79 ms for the pairs (38k FP64 instructions per warp and 32 frequencies;
// eight warps an SM at 255 registers leave the FP64 pipe 35 % busy) and 0.08 ms for the rest.
#include "kr_adjsum.cuh"
#include "kr_hess.cuh"
#include "kr_internal.cuh"
#include "kr_phase.cuh"
#include "kr_prep.cuh"

namespace kr {

constexpr int kHessThreads = 128;
constexpr int kStepVals = 10;  // complex values of a HessStep
constexpr size_t kStepBytes = (size_t)256 << 20;

// ---------------------------------------------------------------------------------------
// Rays
// ---------------------------------------------------------------------------------------
struct HessRaySink {
  bool valid, fs, grow;
  const double2* obs;
  double2* out;   // step values of this (p, omega), value c of step i at out[(i kStepVals + c) n_w]
  double2* seeds; // seed and zeta of this (p, omega)
  int n_w, I;
  const Iface* coef;
  double* acc;
  cd* stage;
  cd sigma;  // sqrt(seed): the adjoint sums are of seed times products of two
  S3 K;
  __device__ cd reflectivity(cd R) {
    sigma = mk(0.0, 0.0);
    if (valid) {
      const double2 o = *obs;
      cd seed = mk(2.0 * (R.x - o.x), -2.0 * (R.y - o.y));
      if (grow) seed = mk(nan(""), nan(""));  // these formulas lose growing phases: no value
      // 1 + Y = 1 / (1 - R) with the free surface
      const cd zeta = fs ? (-2.0 * seed) * recip(1.0 - R) : mk(0.0, 0.0);
      seeds[0] = make_double2(seed.x, seed.y);
      seeds[1] = make_double2(zeta.x, zeta.y);
      sigma = csqrt_any(seed);
    }
    return mk(1.0, 0.0);
  }
  __device__ void top(cd) {}
  __device__ void ray(int i, const Ray& g, const Ray& x, const Ray& wz, const S3& X, cd ea,
                      cd eb) {
    if (valid) {
      const cd v[kStepVals] = {X.a, X.b, X.d, ea, eb, g.a, g.b, K.a, K.b, K.d};
#pragma unroll
      for (int c = 0; c < kStepVals; ++c)
        out[((size_t)i * kStepVals + c) * n_w] = make_double2(v[c].x, v[c].y);
    }
    Ray gs = scale(sigma, g), xs = scale(sigma, x), ws = scale(sigma, wz);
    if (!valid) gs = xs = ws = zero_ray();
    ray_add(gs, xs, ws, stage, acc + (size_t)i * kRayRow);
    if (i < I - 1) K = hess_next_k(K, X, ea, eb, coef[i]);
  }
};

__global__ void __launch_bounds__(kHessThreads, 2)
hess_rays_kernel(int L, const double2* __restrict__ omega, int n_w, int n_wtiles,
                 int free_surface, int seg, int table, const LayerP* __restrict__ lay_all,
                 const Iface* __restrict__ coef_all, const double2* __restrict__ obs, int p0,
                 double2* __restrict__ steps, double2* __restrict__ seeds,
                 cd* __restrict__ sums) {
  constexpr int W = kHessThreads / 32;
  extern __shared__ __align__(16) double s_raw[];
  const int I = L - 1;
  const int jp = blockIdx.x / n_wtiles, ip = p0 + jp;  // slowness within the turn, and overall
  const int tile = blockIdx.x % n_wtiles;
  const int iw = tile * kHessThreads + threadIdx.x;
  const bool valid = iw < n_w;
  const int warp = threadIdx.x >> 5;
  const int nrow = (int)sum_rows(L) * kRayRow;
  double* acc = s_raw;
  cd* stage = reinterpret_cast<cd*>(acc + (size_t)W * nrow);
  Iface* sc = reinterpret_cast<Iface*>(stage + W * kRayStage);
  LayerP* sl = reinterpret_cast<LayerP*>(sc + I);
  cd* s_lo = reinterpret_cast<cd*>(sl + L);
  sums_zero(acc, L, W);
  copy16(sc, coef_all + (size_t)ip * I, sizeof(Iface) * I);
  copy16(sl, lay_all + (size_t)ip * L, sizeof(LayerP) * L);
  __syncthreads();
  cd w = mk(0.0, 0.0);
  if (valid) {
    const double2 wv = omega[iw];
    w = mk(wv.x, wv.y);
  }
  const bool tab = table != 0;
  bool on = ray_line_model(L);  // the tile on the line (and, with a table, its lo entries usable)
  cd* hm = s_lo + ray_lo_values(L) + warp * ray_hm_values(L);
  if (on) {
    const GridLine g = grid_line(omega, n_w);
    if (tab) on = ray_lo_fill(g, L, sl, s_lo);
    if (valid) on &= on_line(g, iw, make_double2(w.x, w.y));
    on = __syncthreads_and(on) != 0;
  }
  const bool use_tab =
      tab && on && ray_hm_fill(omega, n_w, tile * kHessThreads + 32 * warp, L, sl, hm);
  const size_t k = valid ? iw : 0;
  HessRaySink sink;
  sink.valid = valid;
  sink.fs = free_surface != 0;
  sink.grow = phases_grow(w);
  sink.obs = obs + (size_t)ip * n_w + k;
  sink.out = steps + (size_t)jp * I * kStepVals * n_w + k;
  sink.seeds = seeds + 2 * ((size_t)jp * n_w + k);
  sink.n_w = n_w;
  sink.I = I;
  sink.coef = sc;
  sink.acc = acc + (size_t)warp * nrow;
  sink.stage = stage + warp * kRayStage;
  sink.K = S3{mk(0.0, 0.0), mk(0.0, 0.0), mk(0.0, 0.0)};
  if (use_tab)
    adjoint_rays(L, w, free_surface != 0, seg, sc, ray_table(s_lo, hm), sink);
  else
    adjoint_rays(L, w, free_surface != 0, seg, sc, phase_line(on && !tab, omega, n_w, iw, w, sl),
                 sink);
  __syncthreads();
  for (int e = threadIdx.x; e < nrow; e += kHessThreads) {
    double s = acc[e];
    for (int wi = 1; wi < W; ++wi) s += acc[wi * nrow + e];
    acc[e] = s;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < I; i += kHessThreads) {
    cd v[kSumVals];
    ray_row_sums(acc + (size_t)i * kRayRow, v);
    cd* dst = sums + (((size_t)ip * n_wtiles + tile) * I + i) * kSumVals;
    for (int c = 0; c < kSumVals; ++c) dst[c] = v[c];
  }
}

// ---------------------------------------------------------------------------------------
// Pairs
// ---------------------------------------------------------------------------------------
// A block takes 16 frequencies of a slowness at a time; a half-warp takes a layer (lane =
// frequency).  In rounds of eight layers from the half-space up, every half-warp forms its
// layer's vectors, publishes in shared memory what shallower layers read (w, G, A: 4 KB per
// layer; dx: a ring of nine layers, as only the next one up reads it), and after a barrier runs
// its own column of pairs: itself, the layer below, and, with its g^(k) carried down in
// registers, every deeper layer.  Each pair's 16 entries are summed over the half-warp's
// frequencies through a padded tile and added to the block's row of partial sums by reductions
// that nothing waits for (a load, an add and a store per pair stalled each pair on L2).  The
// round's tangents and coefficients (nine interfaces) are staged in the tiles' memory, which the
// pairs need only later: read through L1, of which two blocks leave 12 KB, they missed.
// 16 frequencies per block: two blocks of a 21-layer model fit an SM (108 KB each), so one's
// near stage covers the other's barrier.
constexpr int kPairFreq = 16;
constexpr int kPairGroups = kHessThreads / kPairFreq;  // layers per round
constexpr int kPubVals = 16;                           // w 8, G 4, A 4
constexpr int kDxSlots = kPairGroups + 1;
constexpr int kTileRow = 10;                           // doubles per frequency, 8 used

// Interfaces a round of layers touches, and where their data sits in the tiles' memory.
constexpr int kRoundIfaces = kPairGroups + 1;
constexpr size_t kTileBytes = sizeof(double) * kPairGroups * kPairFreq * kTileRow;
static_assert(kRoundIfaces * (sizeof(ScatTan) + sizeof(HessIface)) <= kTileBytes,
              "a round's tangents and coefficients fit the tiles");

static size_t hess_pairs_smem(int L) {
  return sizeof(cd) * kPairFreq * ((size_t)kPubVals * (L - 1) + 8 * kDxSlots) + kTileBytes;
}
// Layers whose published values fit a block's shared memory (50).
constexpr size_t kHessSmemMax = 227 * 1024;
static bool hess_fits(int L) { return hess_pairs_smem(L) <= kHessSmemMax; }

struct SmemPublisher {
  cd* pub;  // this (layer, frequency): value c at pub[c kPairFreq]
  cd* dx;
  __device__ __forceinline__ void set_w(int j, const Ray& v) {
    pub[(2 * j) * kPairFreq] = v.a;
    pub[(2 * j + 1) * kPairFreq] = v.b;
  }
  __device__ __forceinline__ void set_G(int c, cd v) { pub[(8 + c) * kPairFreq] = v; }
  __device__ __forceinline__ void set_A(int j, cd v) { pub[(12 + j) * kPairFreq] = v; }
  __device__ __forceinline__ void set_dx(int j, const Ray& v) {
    dx[(2 * j) * kPairFreq] = v.a;
    dx[(2 * j + 1) * kPairFreq] = v.b;
  }
};

// Sum over the half-warp of v[c], c < 8: the result for c = lane & 7.  `tile`: the half-warp's
// [16][kTileRow] doubles; `mask`: its lanes.
__device__ __forceinline__ double half_sum8(const double v[8], double* tile, unsigned mask) {
  const int q = threadIdx.x & 15;
  double2* mine = reinterpret_cast<double2*>(tile + q * kTileRow);
#pragma unroll
  for (int c = 0; c < 4; ++c) mine[c] = make_double2(v[2 * c], v[2 * c + 1]);
  __syncwarp(mask);
  const double* col = tile + (q >> 3) * 8 * kTileRow + (q & 7);
  double s = col[0];
#pragma unroll
  for (int r = 1; r < 8; ++r) s += col[r * kTileRow];
  s += __shfl_xor_sync(mask, s, 8);
  __syncwarp(mask);
  return s;
}

__global__ void __launch_bounds__(kHessThreads, 2)
hess_pairs_kernel(int L, const double2* __restrict__ omega, int n_w, int n_wc, int n_chunks,
                  const LayerD* __restrict__ dlay_all, const Iface* __restrict__ coef_all,
                  const ScatTan* __restrict__ tan_all, const double2* __restrict__ steps,
                  const double2* __restrict__ seeds, int p0, double* __restrict__ partial) {
  // the curvature kernel does not read this one's results: it may start when there is room
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(16) cd s_pub[];  // [I][kPubVals][16], [kDxSlots][8][16], tiles
  const int I = L - 1;
  cd* s_dx = s_pub + (size_t)I * kPubVals * kPairFreq;
  double* s_tile = reinterpret_cast<double*>(s_dx + 8 * kDxSlots * kPairFreq);
  const int q = threadIdx.x & 15, h = threadIdx.x >> 4;
  double* tile = s_tile + h * kPairFreq * kTileRow;
  const unsigned mask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  double* part = partial + (size_t)blockIdx.x * (I * (I + 1) / 2) * 16;
  const cd zero = mk(0.0, 0.0);
  for (int chunk = blockIdx.x; chunk < n_chunks; chunk += gridDim.x) {
    const int jp = chunk / n_wc, ip = p0 + jp;
    const int iw = (chunk % n_wc) * kPairFreq + q;
    const bool valid = iw < n_w;
    cd w = zero, seed = zero, zeta = zero;
    if (valid) {
      const double2 a = omega[iw];
      const double2* sz = seeds + 2 * ((size_t)jp * n_w + iw);
      const double2 b = sz[0], c = sz[1];
      w = mk(a.x, a.y);
      seed = mk(b.x, b.y);
      zeta = mk(c.x, c.y);
    }
    const double2* st = steps + (size_t)jp * I * kStepVals * n_w + (valid ? iw : 0);
    auto load = [&](int i, int c) {
      if (!valid) return zero;
      const double2 v = st[((size_t)i * kStepVals + c) * n_w];
      return mk(v.x, v.y);
    };
    // adds the sums of 16 entries (j 4 + k: parameter j of layer l, k of layer m <= l)
    auto store = [&](const double v[16], int l, int m) {
      double* dst = part + ((size_t)(l * (l - 1) / 2 + m - 1)) * 16;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const double s = half_sum8(v + 8 * half, tile, mask);
        // one block and one lane per address, in program order: a fixed order of additions
        if (q < 8) atomicAdd(dst + 8 * half + q, s);
      }
    };
    // the first (deepest) round takes the remainder, where columns are shortest: a round lasts as
    // long as its longest column
    const int first = (I - 1) % kPairGroups + 1;
    for (int base = I, size = first; base >= 1; base -= size, size = kPairGroups) {
      const int l = h < size ? base - h : 0;
      HessOwn own;
      // interfaces i0 .. i0 + kRoundIfaces - 1 of the round's layers (those that exist)
      const int i0 = base - size, ni = min(base, I - 1) - i0 + 1;
      ScatTan* s_tan = reinterpret_cast<ScatTan*>(s_tile);
      HessIface* s_if = reinterpret_cast<HessIface*>(s_tan + kRoundIfaces);
      copy16(s_tan, tan_all + (size_t)ip * I + i0, sizeof(ScatTan) * ni);
      for (int e = threadIdx.x; e < 7 * ni; e += kHessThreads) {
        const int i = e / 7, c = e - 7 * i;  // ru11 .. td22 are entries 3 .. 9 of an Iface
        reinterpret_cast<cd*>(s_if + i)[c] =
            reinterpret_cast<const cd*>(coef_all + (size_t)ip * I + i0 + i)[3 + c];
      }
      __syncthreads();
      if (l >= 1) {
        HessStep lo, up;
        const bool full = l <= I - 1;
        lo.X = full ? S3{load(l - 1, 0), load(l - 1, 1), load(l - 1, 2)} : S3{zero, zero, zero};
        lo.ea = full ? load(l - 1, 3) : zero;
        lo.eb = full ? load(l - 1, 4) : zero;
        lo.g = Ray{load(l - 1, 5), load(l - 1, 6)};
        lo.K = S3{load(l - 1, 7), load(l - 1, 8), load(l - 1, 9)};
        const int u = full ? l : l - 1;  // the half-space has no step below it
        up.X = S3{zero, zero, zero};
        up.ea = up.eb = zero;
        if (l <= I - 2) {
          up.X = S3{load(l, 0), load(l, 1), load(l, 2)};
          up.ea = load(l, 3);
          up.eb = load(l, 4);
        }
        up.g = full ? Ray{load(l, 5), load(l, 6)} : zero_ray();
        up.K = S3{zero, zero, zero};
        SmemPublisher pub{s_pub + (size_t)(l - 1) * kPubVals * kPairFreq + q,
                          s_dx + (l % kDxSlots) * 8 * kPairFreq + q};
        hess_layer(l, I, w, seed, zeta, lo, up, s_if[l - 1 - i0], s_if[u - i0], s_tan[l - 1 - i0],
                   s_tan[u - i0], dlay_all[(size_t)ip * L + l], pub, own);
      }
      __syncthreads();
      if (valid && base - size - h >= 1) {
        // the next round's steps, towards L2 while the pairs run
        const double2* nx = st + (size_t)(base - size - h - 1) * kStepVals * n_w;
#pragma unroll
        for (int c = 0; c < kStepVals; ++c)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + (size_t)c * n_w));
      }
      if (l >= 1) {
        double v[16];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) v[4 * j + k] = k <= j ? own.s[j * (j + 1) / 2 + k] : 0.0;
        store(v, l, l);
        if (l + 1 <= I) {
          const cd* pb = s_pub + (size_t)l * kPubVals * kPairFreq + q;
          const cd* dx = s_dx + ((l + 1) % kDxSlots) * 8 * kPairFreq + q;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const Ray wj = {pb[2 * j * kPairFreq], pb[(2 * j + 1) * kPairFreq]};
            const Ray dj = {dx[2 * j * kPairFreq], dx[(2 * j + 1) * kPairFreq]};
            const cd A = pb[(12 + j) * kPairFreq];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[4 * j + k] = hess_adjacent(wj, dj, A, own, k);
          }
          store(v, l + 1, l);
        }
        Ray g[4] = {own.gn[0], own.gn[1], own.gn[2], own.gn[3]};
        for (int d = l + 2; d <= I; ++d) {
          const cd* pb = s_pub + (size_t)(d - 1) * kPubVals * kPairFreq + q;
          if (d > l + 2) {
            const cd* Gp = pb - (size_t)2 * kPubVals * kPairFreq + 8 * kPairFreq;
            const cd G[4] = {Gp[0], Gp[kPairFreq], Gp[2 * kPairFreq], Gp[3 * kPairFreq]};
#pragma unroll
            for (int k = 0; k < 4; ++k) g[k] = hess_down(G, g[k]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const Ray wj = {pb[2 * j * kPairFreq], pb[(2 * j + 1) * kPairFreq]};
            const cd A = pb[(12 + j) * kPairFreq];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[4 * j + k] = hess_far(wj, A, g[k], own.J[k]);
          }
          store(v, d, l);
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------------------
// Curvature of the coefficients and phases, and the sum of everything
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128)
hess_curvature_kernel(const double* __restrict__ tab, int L, const double* __restrict__ p, int n_p,
                      int n_wtiles, const LayerP* __restrict__ lay, const LayerD* __restrict__ dlay,
                      const cd* __restrict__ sums, double* __restrict__ out) {
  const int I = L - 1;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (size_t)n_p * I * kHessItems) {
    const int item = (int)(t % kHessItems);
    const size_t idx = t / kHessItems;
    const int ip = (int)(idx / I), i = (int)(idx % I);
    cd S[kSumVals];
    const cd* src = sums + ((size_t)ip * n_wtiles * I + i) * kSumVals;
    for (int k = 0; k < kSumVals; ++k) S[k] = src[k];
    for (int u = 1; u < n_wtiles; ++u)
      for (int k = 0; k < kSumVals; ++k) S[k] = S[k] + src[(size_t)u * I * kSumVals + k];
    const LayerP* lp = lay + (size_t)ip * L;
    const LayerD* ld = dlay + (size_t)ip * L;
    LayerD2 d2[2];
    for (int k = 0; k < 2; ++k) d2[k] = layer_derivs2(tab, L, i + k, lp[i + k], ld[i + k]);
    out[t] = hess_curvature(tab, L, i, p[ip], lp, ld, d2, S, item);
  }
  // launched as the pair kernel's programmatic dependent, to fill the SMs as its blocks finish:
  // complete only after it, so that the assembly finds both
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Entry (l, j, m, k), m <= l, of the lower triangle: rows of `partial`, plus the curvature terms
// of the interface(s) and phase the two parameters share.  32 entries x 32 row groups per block:
// each thread's loads are a serial chain through L2.
constexpr int kAsmGroups = 32;
__global__ void __launch_bounds__(32 * kAsmGroups)
hess_assemble_kernel(int I, const double* __restrict__ partial, int n_rows, int n_p,
                     const double* __restrict__ curv, double* __restrict__ H) {
  __shared__ double s[kAsmGroups][33];
  const int n_ent = I * (I + 1) / 2 * 16;
  const int e = blockIdx.x * 32 + (threadIdx.x & 31), grp = threadIdx.x >> 5;
  double t = 0.0;
  int l = 1, m = 1, j = 0, k = 0;
  if (e < n_ent) {
    const int pair = e / 16;
    while (l * (l + 1) / 2 <= pair) ++l;
    m = pair - l * (l - 1) / 2 + 1;
    j = (e >> 2) & 3;
    k = e & 3;
    for (int r = grp; r < n_rows; r += kAsmGroups) t += partial[(size_t)r * n_ent + e];
    int item[3] = {-1, -1, -1}, at[3] = {0, 0, 0};
    auto sym = [](int a, int b) { return a >= b ? a * (a + 1) / 2 + b : b * (b + 1) / 2 + a; };
    if (l == m && k <= j) {
      if (j < 3) {
        item[0] = sym(3 + j, 3 + k);
        at[0] = l - 1;
        if (l <= I - 1) {
          item[1] = sym(j, k);
          at[1] = l;
        }
      }
      item[2] = j == 0 ? 21 : j == 1 && k == 1 ? 23 : j == 3 && k == 0 ? 22 : j == 3 && k == 1 ? 24 : -1;
      at[2] = l - 1;
    } else if (l == m + 1 && j < 3 && k < 3) {
      item[0] = sym(3 + j, k);
      at[0] = m;
    }
    for (int c = 0; c < 3; ++c)
      if (item[c] >= 0)
        for (int r = grp; r < n_p; r += kAsmGroups)
          t += curv[((size_t)r * I + at[c]) * kHessItems + item[c]];
  }
  s[grp][threadIdx.x & 31] = t;
  __syncthreads();
  if (grp != 0 || e >= n_ent || (l == m && k > j)) return;
  for (int r = 1; r < kAsmGroups; ++r) t += s[r][threadIdx.x];
  const int n = 4 * I, row = j * I + l - 1, col = k * I + m - 1;
  H[(size_t)row * n + col] = t;
  H[(size_t)col * n + row] = t;
}

static size_t a256s(size_t x) { return (x + 255) & ~(size_t)255; }

constexpr int kHessRows = 148 * 2;  // resident blocks of the pair kernel, hence rows of partial sums

struct HessWs {
  LayerP* lay;
  LayerD* dlay;
  Iface* coef;
  ScatTan* tan;
  double2* steps;   // [turn][I][kStepVals][n_w]
  double2* seeds;   // [turn][n_w][2]
  cd* sums;         // [n_p][n_wtiles][I][12]
  double* curv;     // [n_p][I][kHessItems]
  double* partial;  // [kHessRows][pairs][16]
  int turn;         // slownesses per turn
  size_t bytes;
};

static HessWs hess_ws(void* base, int L, int n_p, int n_w) {
  HessWs w;
  const size_t I = L - 1, np = n_p, nw = n_w;
  const size_t n_wtiles = (nw + kHessThreads - 1) / kHessThreads;
  const size_t per = sizeof(double2) * nw * (I * kStepVals + 2);
  size_t turn = kStepBytes / per;
  if (turn < 1) turn = 1;
  if (turn > np) turn = np;
  w.turn = (int)turn;
  unsigned char* b = static_cast<unsigned char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* r = b + off;
    off = a256s(off + bytes);
    return r;
  };
  w.lay = reinterpret_cast<LayerP*>(take(sizeof(LayerP) * np * L));
  w.dlay = reinterpret_cast<LayerD*>(take(sizeof(LayerD) * np * L));
  w.coef = reinterpret_cast<Iface*>(take(sizeof(Iface) * np * I));
  w.tan = reinterpret_cast<ScatTan*>(take(sizeof(ScatTan) * np * I));
  w.steps = reinterpret_cast<double2*>(take(sizeof(double2) * turn * I * kStepVals * nw));
  w.seeds = reinterpret_cast<double2*>(take(sizeof(double2) * turn * nw * 2));
  w.sums = reinterpret_cast<cd*>(take(sizeof(cd) * np * n_wtiles * I * kSumVals));
  w.curv = reinterpret_cast<double*>(take(sizeof(double) * np * I * kHessItems));
  w.partial = reinterpret_cast<double*>(take(sizeof(double) * kHessRows * (I * (I + 1) / 2) * 16));
  w.bytes = off;
  return w;
}

}  // namespace kr

using namespace kr;

extern "C" size_t kr_misfit_hessian_workspace_bytes(int32_t n_layers, int32_t n_p, int32_t n_w) {
  if (n_layers < 2 || n_layers > kMaxLayers || n_p <= 0 || n_w <= 0 || !hess_fits(n_layers))
    return 0;
  return hess_ws(nullptr, n_layers, n_p, n_w).bytes;
}

extern "C" kr_status kr_misfit_hessian(const double* layers, int32_t n_layers, const double* p,
                                       int32_t n_p, const double* omega, int32_t n_w,
                                       uint32_t flags, const double* R_obs, double* H,
                                       void* workspace, size_t workspace_bytes, void* stream) {
  const int L = n_layers, I = L - 1;
  if (n_p < 0 || n_w < 0 || (flags & ~KR_FREE_SURFACE) || !H) return KR_ERR_INVALID_ARGUMENT;
  if (L < 2) return KR_ERR_INVALID_MODEL;
  if (L > kMaxLayers) return KR_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  if (n_p == 0 || n_w == 0) {  // whatever the depth: the sum over nothing
    const cudaError_t e = cudaMemsetAsync(H, 0, sizeof(double) * 16 * (size_t)I * I, st);
    if (e != cudaSuccess) set_last_error("kr_misfit_hessian: memset", e);
    return cuda_status(e);
  }
  if (!hess_fits(L)) return KR_ERR_TOO_LARGE;
  if (!layers || !p || !omega || !R_obs) return KR_ERR_INVALID_ARGUMENT;
  if (!aligned16(omega) || !aligned16(R_obs)) return KR_ERR_INVALID_ARGUMENT;
  const HessWs w = hess_ws(workspace, L, n_p, n_w);
  if (!workspace || workspace_bytes < w.bytes) return KR_ERR_WORKSPACE;
  const int n_wtiles = (n_w + kHessThreads - 1) / kHessThreads;
  const int n_wc = (n_w + kPairFreq - 1) / kPairFreq;
  const size_t n_curv = (size_t)n_p * I * kHessItems;
  if ((size_t)n_p * n_wc > 0x7fffffffULL ||
      (n_curv + 127) / 128 > 0x7fffffffULL)
    return KR_ERR_TOO_LARGE;
  const double2* w2 = reinterpret_cast<const double2*>(omega);
  kr_status s = launch_prep(layers, L, p, n_p, w.lay, w.dlay, w.coef, w.tan, st,
                            "kr_misfit_hessian: layers and interfaces");
  if (s != KR_OK) return s;
  const int table = ray_table_model(L) ? 1 : 0;
  const size_t rs = raysum_smem_bytes(L, kHessThreads / 32) + prologue_smem_bytes(L) +
                    (table ? ray_table_bytes(L, kHessThreads / 32) : 0);
  const size_t ps = hess_pairs_smem(L);
  static SmemLimit rlim, plim;
  if (rs > 48 * 1024) {
    s = raise_smem_limit((const void*)hess_rays_kernel, rs, rlim, "kr_misfit_hessian: ray smem");
    if (s != KR_OK) return s;
  }
  if (ps > 48 * 1024) {
    s = raise_smem_limit((const void*)hess_pairs_kernel, ps, plim, "kr_misfit_hessian: pair smem");
    if (s != KR_OK) return s;
  }
  const int seg = checkpoint_spacing(I > 1 ? I - 1 : 1);
  const int rows = n_wc * (long long)w.turn < kHessRows ? n_wc * w.turn : kHessRows;
  const int n_ent = I * (I + 1) / 2 * 16;
  const cudaError_t me = cudaMemsetAsync(w.partial, 0, sizeof(double) * n_ent * (size_t)rows, st);
  if (me != cudaSuccess) {
    set_last_error("kr_misfit_hessian: memset", me);
    return KR_ERR_CUDA;
  }
  for (int p0 = 0; p0 < n_p; p0 += w.turn) {
    const int np = n_p - p0 < w.turn ? n_p - p0 : w.turn;
    hess_rays_kernel<<<(unsigned)(np * n_wtiles), kHessThreads, rs, st>>>(
        L, w2, n_w, n_wtiles, (flags & KR_FREE_SURFACE) ? 1 : 0, seg, table, w.lay, w.coef,
        reinterpret_cast<const double2*>(R_obs), p0, w.steps, w.seeds, w.sums);
    s = check_launch("kr_misfit_hessian: rays");
    if (s != KR_OK) return s;
    const int chunks = np * n_wc;
    hess_pairs_kernel<<<(unsigned)(chunks < rows ? chunks : rows), kHessThreads, ps, st>>>(
        L, w2, n_w, n_wc, chunks, w.dlay, w.coef, w.tan, w.steps, w.seeds, p0, w.partial);
    s = check_launch("kr_misfit_hessian: pairs");
    if (s != KR_OK) return s;
  }
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)((n_curv + 127) / 128));
  lc.blockDim = dim3(128);
  lc.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  const cudaError_t ce = cudaLaunchKernelEx(&lc, hess_curvature_kernel, layers, L, p, n_p, n_wtiles,
                                            (const LayerP*)w.lay, (const LayerD*)w.dlay,
                                            (const cd*)w.sums, w.curv);
  if (ce != cudaSuccess) {
    set_last_error("kr_misfit_hessian: curvature", ce);
    return KR_ERR_CUDA;
  }
  hess_assemble_kernel<<<(unsigned)((n_ent + 31) / 32), 32 * kAsmGroups, 0, st>>>(I, w.partial, rows, n_p,
                                                                      w.curv, H);
  return check_launch("kr_misfit_hessian: assemble");
}
