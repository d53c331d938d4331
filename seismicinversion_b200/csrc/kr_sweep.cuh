// The forward sweep of one slowness over a uniform frequency grid, warp by warp, shared by the
// per-model and the batched forward kernels (so that both give the same bits) and, with its own
// form of the recursion, by the global-matrix kernel.
//
// What bounds it is the FP64 pipe: ~115 FP64 instructions per (omega, p, interface) in
// kennett_step_x when the squared and mixed phase factors P = ea^2, Q = eb^2, S = ea eb come
// from a table.  The table holds, for the phases exp(omega c) with c = i eta h and i neta h of
// every layer above the half-space, lo[j] = exp(j delta c), j < 16, and mid[m] = exp(16 m delta c),
// m < 8, as their squares and product; a warp forms hi = exp(omega_{128 u} c) of its tile u (again
// squares and product) times the mid entries of its own frequencies once per pass (hm), so a
// lookup is one complex product of two shared-memory reads.  P, Q and S come from the same two
// exponentials so that S^2 = P Q holds to a few roundings whatever the rounding of omega c: models
// near a pole amplify a mismatch (exp of 2 c and of the sums instead: global-matrix R of the
// 5-layer model off by 1.8 times as much at 0.7 to 1 s/km).  Models too deep for three phases per layer in shared memory
// tabulate ea and eb alone (two lookups and three more products per step); models deeper still
// evaluate exponentials directly, as do tiles that are off the grid's line (kr_phase.cuh).
//
// A lane sweeps F frequencies at once (the kernels use 1; 2 halves the reads of the 17
// coefficients per step but costs more registers than it gains, kr_forward.cu).
#pragma once

#include "kr_phase.cuh"

namespace kr {

// Phases per layer of a tabulating model: 3 (P, Q, S) up to kPqsLayers layers, where a block of
// four warps (58 KB at 30 layers, 50 KB for one with a pass) fits three or four times on an SM; 2 (ea, eb) up to kPairLayers, where
// a block of eight warps (113 KB at 66) fits twice: 193 x 1501 of a 64-layer model takes 230 us
// against 351 with direct exponentials; 0 beyond.  Every forward kernel applies this rule to
// the model, so a model's phases round alike everywhere.
constexpr int kPqsLayers = 30;
constexpr int kPairLayers = 66;
__host__ __device__ inline int sweep_phases(int n_layers) {
  return n_layers <= kPqsLayers ? 3 : n_layers <= kPairLayers ? 2 : 0;
}
// The same two phases' values without a table: the lanes of a warp form its entries step by step
// (SweepLanes).
constexpr int kLanePhases = 1;

// Shared memory of one slowness (layer terms and roots, interface coefficients, lo / mid
// entries) and of
// one warp (its hm products) for NPH phases per layer and F frequencies per lane.  Without a table
// the roots lie where the coefficients come to lie, but for the last layer's.
__host__ __device__ inline size_t sweep_slowness_bytes(int n_layers, int nph) {
  return prologue_smem_bytes(n_layers) + sizeof(LayerRoots) * (nph > 1 ? n_layers : 1) +
         (nph > 1 ? sizeof(cd) * kPhHead * nph * (size_t)(n_layers - 1) : 0);
}
__host__ __device__ inline size_t sweep_warp_bytes(int n_layers, int nph, int F) {
  return sizeof(cd) * 2 * F * (nph == kLanePhases ? 2 : nph) * (size_t)(n_layers - 1);
}

// Exponent `id` (2 l + k) of a model: i eta h of layer l, or i neta h.
__device__ __forceinline__ cd sweep_exponent(const LayerP* lay, int id) {
  const LayerP& lp = lay[id >> 1];
  return id & 1 ? lp.cb : lp.ca;
}

__device__ __forceinline__ bool phase_usable(cd v) {
  return fabs(v.x) <= kPhMaxMag && fabs(v.y) <= kPhMaxMag;
}

// Entry j (lo, then mid) of every phase of layer l of a slowness's table; returns whether they are
// usable.
template <int NPH>
__device__ __forceinline__ bool sweep_table_entry(const GridLine& g, const LayerP* lay, int l,
                                                  int j, cd* tab) {
  const cd z = (double)(j < kPhLo ? j : (j - kPhLo) * kPhLo) * g.d;
  const cd a = cexp_(z * lay[l].ca), b = cexp_(z * lay[l].cb);
  cd* t = tab + (size_t)NPH * l * kPhHead + j;
  const cd u = NPH == 3 ? a * a : a, v = NPH == 3 ? b * b : b;
  t[0] = u;
  t[kPhHead] = v;
  if (NPH == 3) t[2 * kPhHead] = a * b;
  return phase_usable(u) && phase_usable(v);
}

// The prologue's two stages out of line: one compiled body per kernel file, called by every
// kernel that must agree bit for bit, and no register pressure on the sweep around it.  Stage 1,
// a thread per (layer, P or S): terms and square root; stage 2, a thread per interface: the
// coefficients, a chain of complex products once the roots are there.
static __device__ __noinline__ void layer_store(const double* tab, int L, int l, int half,
                                                double p, LayerP* lay, LayerRoots* roots) {
  if (half == 0) {
    layer_terms_p(tab, L, l, p, *lay);
    roots->eta = csqrt(lay->eta);
  } else {
    layer_terms_s(tab, L, l, p, *lay);
    roots->neta = csqrt(lay->neta);
  }
}
static __device__ __noinline__ void interface_store(double p, int i, const LayerP* lay,
                                                    const LayerRoots* up, const LayerRoots* lo,
                                                    Iface* out) {
  *out = interface_coeffs(p, i, lay[i], lay[i + 1], *up, *lo);
}

// Phase factors of F frequencies of one lane from the table.
template <int NPH, int F>
struct SweepTable {
  const cd* lo;  // the lane's lo entry of phase 0
  const cd* hm;  // the lane's first hm product of phase 0 (frequency f: + 2 f)
  __device__ __forceinline__ void pqs(int l, cd P[F], cd Q[F], cd S[F]) const {
    const cd* a = lo + (size_t)(NPH * l) * kPhHead;
    const cd* b = hm + (size_t)(NPH * l) * 2 * F;
    const cd l0 = a[0], l1 = a[kPhHead];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const cd u = b[2 * f] * l0, v = b[2 * F + 2 * f] * l1;
      if (NPH == 3) {
        P[f] = u;
        Q[f] = v;
        S[f] = b[4 * F + 2 * f] * a[2 * kPhHead];
      } else {
        P[f] = u * u;
        Q[f] = v * v;
        S[f] = u * v;
      }
    }
  }
  __device__ __forceinline__ void ocean(cd E[F]) const {  // e0^2
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const cd u = hm[2 * f] * lo[0];
      E[f] = NPH == 3 ? u : u * u;
    }
  }
};

// Direct exponentials of one frequency.
struct SweepDirect {
  cd w;
  const LayerP* lay;
  __device__ __forceinline__ void pqs(int l, cd P[1], cd Q[1], cd S[1]) const {
    const cd a = cexp_(w * lay[l].ca), b = cexp_(w * lay[l].cb);
    P[0] = a * a;
    Q[0] = b * b;
    S[0] = a * b;
  }
  __device__ __forceinline__ void ocean(cd E[1]) const {
    const cd a = cexp_(w * lay[0].ca);
    E[0] = a * a;
  }
};

// Phase factors ea, eb of the table, bit for bit, without its lo entries in memory: lane 16 q + j forms
// entry j of phase q (P, S) of the layer at hand, and shuffles hand the entries round.  One exponential
// a lane and step (SweepDirect: two), and of shared memory only the warp's hm products: where a
// slowness has few passes, its table (three times the rest of its data) would keep other slownesses
// off the SM (forward_plan).
struct SweepLanes {
  cd zlo;        // the lane's lo entry's exponent over c
  const cd* hm;  // the lane's first hm product of phase 0
  const LayerP* lay;
  static __device__ __forceinline__ cd from(cd v, int lane) {
    return mk(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
  }
  __device__ __forceinline__ SweepLanes(cd d, const cd* h, const LayerP* l)
      : zlo((double)(threadIdx.x & 15) * d), hm(h), lay(l) {}
  __device__ __forceinline__ void pqs(int l, cd P[1], cd Q[1], cd S[1]) const {
    const int lane = threadIdx.x & 31;
    const cd lo = cexp_(zlo * ((lane & 16) ? lay[l].cb : lay[l].ca));
    const cd u = hm[4 * l] * from(lo, lane & 15), v = hm[4 * l + 2] * from(lo, 16 + (lane & 15));
    P[0] = u * u;
    Q[0] = v * v;
    S[0] = u * v;
  }
  __device__ __forceinline__ void ocean(cd E[1]) const {
    const cd u = hm[0] * cexp_(zlo * lay[0].ca);
    E[0] = u * u;
  }
};

// Whether all lo and mid entries of a phase are usable: the exponentials themselves only where their
// size is not plain (below e^200, 1e87).
__device__ __forceinline__ bool phase_table_usable(const GridLine& g, cd c) {
  if ((double)((kPhMid - 1) * kPhLo) * (g.d * c).x <= 200.0) return true;
  bool ok = true;
  for (int j = 0; j < kPhHead; ++j)
    ok &= phase_usable(cexp_(((double)(j < kPhLo ? j : (j - kPhLo) * kPhLo) * g.d) * c));
  return ok;
}

// The Kennett recursion as a form of the sweep: its interface coefficients, formed once per
// (slowness, interface), and the upward sweep of F frequencies, giving R at the surface.
struct KennettForm {
  typedef Iface Coef;
  static __device__ __forceinline__ void store(double p, int i, const LayerP* lay,
                                               const LayerRoots* up, const LayerRoots* lo,
                                               Coef* out) {
    interface_store(p, i, lay, up, lo, out);
  }
  template <int F, class Ph>
  static __device__ __forceinline__ void sweep(int n_layers, const Coef* coef, const Ph& ph,
                                               bool fs, cd R[F]) {
    const int I = n_layers - 1;
    M2 r[F];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      r[f].a = coef[I - 1].rd11;
      r[f].b = coef[I - 1].rd12;
      r[f].d = coef[I - 1].rd22;
    }
    cd P[F], Q[F], S[F], rpp[F], E[F];
#pragma unroll 1
    for (int i = I - 2; i >= 1; --i) {
      ph.pqs(i + 1, P, Q, S);
#pragma unroll
      for (int f = 0; f < F; ++f) {
        cd x11, x12, x22;
        r[f] = kennett_step_x(r[f], P[f], Q[f], S[f], coef[i], x11, x12, x22);
      }
    }
    if (I > 1) ph.pqs(1, P, Q, S);
    ph.ocean(E);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      rpp[f] = I > 1 ? kennett_last_step_pp(r[f], P[f], Q[f], S[f], coef[0]) : r[f].a;
      R[f] = pp_surface2(rpp[f], E[f], fs);
    }
  }
};

// The two kinds of sweep out of line, so that the hot loop's registers are its own: inlined
// next to the exponentials and the task bookkeeping it spilled inside the loop.
template <int F>
struct SweepOut {
  cd R[F];
};
template <class Form, int NPH, int F>
__device__ __noinline__ SweepOut<F> sweep_table(int n_layers, const typename Form::Coef* coef,
                                                const cd* lo, const cd* hm, bool fs) {
  SweepOut<F> o;
  Form::template sweep<F>(n_layers, coef, SweepTable<NPH, F>{lo, hm}, fs, o.R);
  return o;
}
template <class Form>
__device__ __noinline__ cd sweep_lanes(int n_layers, const typename Form::Coef* coef, cd d,
                                       const cd* hm, const LayerP* lay, bool fs) {
  cd R[1];
  Form::template sweep<1>(n_layers, coef, SweepLanes(d, hm, lay), fs, R);
  return R[0];
}
template <class Form>
__device__ __noinline__ cd sweep_direct(int n_layers, const typename Form::Coef* coef,
                                        const LayerP* lay, cd w, bool fs) {
  cd R[1];
  Form::template sweep<1>(n_layers, coef, SweepDirect{w, lay}, fs, R);
  return R[0];
}

// Tiles whose start and verdict a block keeps in shared memory at once.
constexpr int kSweepTiles = 66;
struct SweepTiles {
  double2 w0[kSweepTiles];        // the tile's first frequency
  unsigned char off[kSweepTiles]; // 1: the tile leaves the grid's line
};

// Starts and verdicts of tiles [u0, u0 + n), the block's warps taking tiles in turn; returns whether
// one of this warp's is on the line.  All threads call it; the caller synchronises.  Where no tile of
// the block is, no table is built.
__device__ __forceinline__ bool sweep_tiles_check(const double2* __restrict__ omega, int n_w,
                                                  const GridLine& g, int u0, int n,
                                                  SweepTiles& t) {
  const int lane = threadIdx.x & 31;
  bool any = false;
  for (int v = threadIdx.x >> 5; v < n; v += blockDim.x >> 5) {
    bool off = false;
#pragma unroll
    for (int q = 0; q < kPhTile / 32; ++q) {
      const int k = (u0 + v) * kPhTile + 32 * q + lane;
      if (k >= n_w) continue;
      const double2 w = omega[k];
      const double m = (double)k;
      if (q == 0 && lane == 0) t.w0[v] = w;
      off |= !(fabs(w.x - fma(m, g.d.x, g.w0.x)) <= g.tol && fabs(w.y - fma(m, g.d.y, g.w0.y)) <= g.tol);
    }
    off = __any_sync(0xffffffffu, off);
    if (lane == 0) t.off[v] = off ? 1 : 0;
    any |= !off;
  }
  return any;
}

// One warp: passes [pass0, pass1) of tile u (pass q: the 32 F consecutive frequencies from
// 128 u + 32 F q), frequencies outside [k_lo, k_hi) skipped.  `w0`: the tile's first frequency;
// `use`: whether the tile and the slowness's lo / mid entries `tab` may be used (NPH > 0); hm:
// the warp's scratch.  The tile's hi entries are evaluated once and stay in registers.
template <class Form, int NPH, int F>
__device__ __forceinline__ void sweep_tile(const double2* __restrict__ omega, double2 w0, int u,
                                           int pass0, int pass1, int k_lo, int k_hi, int n_layers,
                                           const LayerP* lay, const typename Form::Coef* coef,
                                           const cd* tab, bool use, cd* hm, bool fs, double2* __restrict__ Rp) {
  const int lane = threadIdx.x & 31;
  constexpr int N = NPH > 0 ? NPH : 1;
  constexpr int kDeepest = NPH == 3 ? kPqsLayers : kPairLayers;
  constexpr int kHi = (2 * (kDeepest - 1) + 31) / 32;
  const int n_exp = 2 * (n_layers - 1);
  // lanes take the exponents in turn; a layer's two lie in neighbouring lanes, which exchange them
  // for the product (formed alike by both, which then share its hm entries)
  cd hi[kHi], hs[NPH == 3 ? kHi : 1];
  if (NPH > 0 && use) {
    bool bad = false;
#pragma unroll
    for (int r = 0; r < kHi; ++r) {
      if (32 * r >= n_exp) break;
      const int id = 32 * r + lane;
      cd e = mk(0.0, 0.0);
      if (id < n_exp) e = cexp_(mk(w0.x, w0.y) * sweep_exponent(lay, id));
      if (NPH == 3) {
        const cd o = mk(__shfl_xor_sync(0xffffffffu, e.x, 1), __shfl_xor_sync(0xffffffffu, e.y, 1));
        hs[r] = (lane & 1) ? o * e : e * o;
        e = e * e;
      }
      hi[r] = e;
      bad |= !phase_usable(e);
    }
    use = !__any_sync(0xffffffffu, bad);
  }
  for (int pass = pass0; pass < pass1; ++pass) {
    const int kb = u * kPhTile + pass * 32 * F;
    if (kb >= k_hi || kb + 32 * F <= k_lo) continue;
    if (NPH > 0 && use) {
#pragma unroll
      for (int r = 0; r < kHi; ++r) {
        const int id = 32 * r + lane;
        if (id < n_exp) {
          const int ph = NPH == 3 ? 3 * (id >> 1) + (id & 1) : id;
          const cd* mid = tab + ph * kPhHead + kPhLo + pass * 2 * F;
#pragma unroll
          for (int m = 0; m < 2 * F; ++m) hm[ph * 2 * F + m] = hi[r] * mid[m];
          if (NPH == 3) {
            const int ps = 3 * (id >> 1) + 2;
            const cd* mids = tab + ps * kPhHead + kPhLo + pass * 2 * F;
#pragma unroll
            for (int m = 0; m < F; ++m) {
              const int k = 2 * m + (id & 1);
              hm[ps * 2 * F + k] = hs[r] * mids[k];
            }
          }
        }
      }
      __syncwarp();
      const SweepOut<F> o = sweep_table<Form, N, F>(n_layers, coef, tab + (lane & (kPhLo - 1)),
                                                    hm + (lane >> 4), fs);
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const int k = kb + 32 * f + lane;
        if (k >= k_lo && k < k_hi) Rp[k] = make_double2(o.R[f].x, o.R[f].y);
      }
      __syncwarp();  // hm is read before the next pass overwrites it
      continue;
    }
    for (int f = 0; f < F; ++f) {
      const int k = kb + 32 * f + lane;
      if (k < k_lo || k >= k_hi) continue;
      const double2 wv = omega[k];
      const cd R = sweep_direct<Form>(n_layers, coef, lay, mk(wv.x, wv.y), fs);
      Rp[k] = make_double2(R.x, R.y);
    }
  }
}

// The same for phases formed by the lanes (passes of 32 frequencies).
template <class Form>
__device__ __forceinline__ void sweep_tile_lanes(const double2* __restrict__ omega, const GridLine& g,
                                                 double2 w0, int u, int pass0, int pass1, int k_lo,
                                                 int k_hi, int n_layers, const LayerP* lay,
                                                 const typename Form::Coef* coef, bool use, cd* hm,
                                                 bool fs, double2* __restrict__ Rp) {
  const int lane = threadIdx.x & 31;
  constexpr int kHi = (2 * (kPairLayers - 1) + 31) / 32;
  const int n_exp = 2 * (n_layers - 1);
  cd hi[kHi];
  if (use) {
    bool ok = true;
#pragma unroll
    for (int r = 0; r < kHi; ++r) {
      const int id = 32 * r + lane;
      if (id >= n_exp) break;
      hi[r] = cexp_(mk(w0.x, w0.y) * sweep_exponent(lay, id));
      ok &= phase_usable(hi[r]);
    }
    use = __all_sync(0xffffffffu, ok);
  }
  for (int pass = pass0; pass < pass1; ++pass) {
    const int kb = u * kPhTile + pass * 32, k = kb + lane;
    if (kb >= k_hi || kb + 32 <= k_lo) continue;
    const bool valid = k >= k_lo && k < k_hi;
    cd R;
    if (use) {
#pragma unroll
      for (int r = 0; r < kHi; ++r) {
        const int id = 32 * r + lane;
        if (id >= n_exp) break;
        const cd c = sweep_exponent(lay, id);
#pragma unroll
        for (int m = 0; m < 2; ++m)
          hm[2 * id + m] = hi[r] * cexp_(((double)((2 * pass + m) * kPhLo) * g.d) * c);
      }
      __syncwarp();
      R = sweep_lanes<Form>(n_layers, coef, g.d, hm + (lane >> 4), lay, fs);
      __syncwarp();  // hm is read before the next pass overwrites it
    } else if (valid) {
      const double2 wv = omega[k];
      R = sweep_direct<Form>(n_layers, coef, lay, mk(wv.x, wv.y), fs);
    }
    if (valid) Rp[k] = make_double2(R.x, R.y);
  }
}

}  // namespace kr
