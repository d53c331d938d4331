// The forward sweep kernel and its launch, for any form of the recursion (kr_sweep.cuh).
//
// A block takes G consecutive slownesses and a range of 128-frequency tiles.  Its prologue puts
// the layer terms, the interface coefficients and the phase tables of all G slownesses into
// shared memory; then its warps take tiles of 128 frequencies (or, where those are few, passes of
// 32 F) in turn, each running the whole bottom-up sweep with the recursion's state in registers,
// with no block barrier.
#pragma once

#include <math.h>

#include "kr_sweep.cuh"

namespace kr {

template <class Form, int NPH, int F, int W, int MINB>
__global__ void __launch_bounds__(32 * W, MINB)
sweep_kernel(const double* __restrict__ tab, int L, const double* __restrict__ p, int n_p,
                    const double2* __restrict__ omega, int n_w, int n_wtiles, int G,
                    int tile_groups, int tiles_per_group, int passes, int free_surface,
                    double2* __restrict__ R) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SweepTiles s_tiles;
  __shared__ unsigned s_bad;  // bit g: slowness g's table has an unusable entry
  constexpr bool kTable = NPH > 1;
  constexpr int N = kTable ? NPH : 2;
  const int I = L - 1;
  const int ip0 = (blockIdx.x / tile_groups) * G;
  const int ng = min(G, n_p - ip0);
  const int t0 = (blockIdx.x % tile_groups) * tiles_per_group;
  const int t1 = min(n_wtiles, t0 + tiles_per_group);
  LayerP* s_lay = reinterpret_cast<LayerP*>(smem);
  typedef typename Form::Coef Coef;
  static_assert(sizeof(Coef) <= sizeof(Iface), "sweep_slowness_bytes covers the form");
  static_assert(sizeof(Coef) >= sizeof(LayerRoots), "a layer's roots fit a coefficient's place");
  Coef* s_coef = reinterpret_cast<Coef*>(s_lay + (size_t)G * L);
  LayerRoots* s_root = reinterpret_cast<LayerRoots*>(s_coef + (size_t)G * I);
  // Roots of layer l of slowness g: with a table, an array; without, where coefficient l comes to lie
  // (the last layer's in the array), which saves the deepest models their second block.
  auto root = [&](int g, int l) {
    if (kTable) return s_root + g * L + l;
    return l < I ? reinterpret_cast<LayerRoots*>(s_coef + g * I + l) : s_root + g;
  };
  cd* s_tab = reinterpret_cast<cd*>(s_root + (size_t)G * (kTable ? L : 1));
  const int n_ent = kTable ? NPH * I * kPhHead : 0;  // table entries of one slowness
  cd* s_hm = s_tab + (size_t)G * n_ent;
  if (threadIdx.x == 0) s_bad = 0u;
  for (int e = threadIdx.x; e < 2 * ng * L; e += 32 * W) {
    const int half = e >= ng * L ? 1 : 0, j = e - half * ng * L;
    layer_store(tab, L, j % L, half, p[ip0 + j / L], s_lay + j, root(j / L, j % L));
  }
  const GridLine line = grid_line(omega, n_w);
  bool on = NPH > 0 && sweep_tiles_check(omega, n_w, line, t0, t1 - t0, s_tiles);
  on = __syncthreads_or(on) != 0;
  if (kTable) {
    for (int e = threadIdx.x; e < ng * I; e += 32 * W) {
      const int g = e / I, i = e - g * I;
      Form::store(p[ip0 + g], i, s_lay + g * L, root(g, i), root(g, i + 1), s_coef + e);
    }
  } else {
    // in rounds: every thread takes its two roots before any writes a coefficient over them
    for (int e0 = 0; e0 < ng * I; e0 += 32 * W) {
      const int e = e0 + threadIdx.x, g = e / I, i = e - g * I;
      const bool have = e < ng * I;
      LayerRoots up, lo;
      if (have) {
        up = *root(g, i);
        lo = *root(g, i + 1);
      }
      __syncthreads();
      if (have) Form::store(p[ip0 + g], i, s_lay + g * L, &up, &lo, s_coef + e);
    }
  }
  if (NPH > 0 && on) {
    unsigned bad = 0u;
    if (kTable) {
      for (int e = threadIdx.x; e < ng * I * kPhHead; e += 32 * W) {
        const int gl = e / kPhHead, g = gl / I;
        if (!sweep_table_entry<N>(line, s_lay + g * L, gl - g * I, e - gl * kPhHead,
                                  s_tab + (size_t)g * n_ent))
          bad |= 1u << g;
      }
    } else {
      for (int e = threadIdx.x; e < ng * 2 * I; e += 32 * W) {
        const int g = e / (2 * I);
        if (!phase_table_usable(line, sweep_exponent(s_lay + g * L, e - g * 2 * I))) bad |= 1u << g;
      }
    }
    if (bad) atomicOr(&s_bad, bad);
  }
  __syncthreads();
  const unsigned bad = s_bad;
  const int warp = threadIdx.x >> 5;
  cd* hm = s_hm + (size_t)warp * 2 * F * (NPH == kLanePhases ? 2 : NPH) * I;
  // tasks: (slowness, tile, `passes` of the tile's passes); single passes: those with frequencies
  const int parts = kPhTile / (32 * F) / passes;
  const int per_slowness = parts == 1 ? t1 - t0
                                      : min((t1 - t0) * parts, (n_w - 1) / (32 * F) + 1 - t0 * parts);
  for (int t = warp; t < ng * per_slowness; t += W) {
    const int g = t / per_slowness, q = t - g * per_slowness;
    const int v = q / parts, pass = (q - v * parts) * passes;
    const bool use = NPH > 0 && s_tiles.off[v] == 0 && ((bad >> g) & 1u) == 0u;
    const double2 w0 = NPH > 0 ? s_tiles.w0[v] : make_double2(0.0, 0.0);
    double2* Rp = R + (size_t)(ip0 + g) * n_w;
    if (NPH == kLanePhases)
      sweep_tile_lanes<Form>(omega, line, w0, t0 + v, pass, pass + passes, 0, n_w, L,
                             s_lay + g * L, s_coef + g * I, use, hm, free_surface != 0, Rp);
    else
      sweep_tile<Form, kTable ? NPH : 0, F>(omega, w0, t0 + v, pass, pass + passes, 0, n_w, L,
                                            s_lay + g * L, s_coef + g * I, s_tab + (size_t)g * n_ent,
                                            use, hm, free_surface != 0, Rp);
  }
}

// Dynamic shared memory of a block of W warps and G slownesses of n_pass passes: a warp has hm products
// only where it has a task.
static size_t sweep_block_bytes(int L, int nph, int W, int F, int G, int n_pass) {
  const int warps = G * n_pass < W ? G * n_pass : W;
  return G * sweep_slowness_bytes(L, nph) + warps * sweep_warp_bytes(L, nph, F);
}

// How many slownesses a block takes (G) and into how many groups their tiles are split: the
// pair with the least estimated time, waves x (prologue + sweeps of a block).  The prologue is
// a latency (layer terms, then coefficients: ~6 us whatever G) plus its table entries, a block's
// sweeps take ~0.5 us per 128 (omega, p, interface) triples of four resident blocks; small
// models and short grids get several slownesses per block, which shares the latency, large
// ones a slowness per block and, with few slownesses, several blocks per slowness.
// Each tile is one warp's task, or, where that leaves warps without work, each pass.
struct ForwardSplit {
  int G, groups, tiles, passes;
};

static ForwardSplit forward_split(long long n_p, int n_wtiles, int L, int nph, int F, int W,
                                  int resident, size_t smem_max, int n_pass) {
  ForwardSplit best{1, 1, n_wtiles, 1};
  double best_cost = 1e300;
  for (int G = 1; G <= 16; ++G) {
    if (G > 1 && (sweep_block_bytes(L, nph, W, F, G, n_pass) > smem_max || G > n_p)) break;
    for (int groups = 1; groups < 2 * n_wtiles; groups *= 2) {
      const int tiles = (n_wtiles + groups - 1) / groups;
      if (tiles > kSweepTiles) continue;
      const long long blocks = ((n_p + G - 1) / G) * groups;
      const double waves = (double)((blocks + 148LL * resident - 1) / (148LL * resident));
      const double cost = waves * (6.0 + G * (L - 1) * (0.05 * nph + 0.5 * tiles));
      if (cost < 0.97 * best_cost) {
        best_cost = cost;
        best = ForwardSplit{G, groups, tiles, 1};
      }
    }
  }
  best.groups = (n_wtiles + best.tiles - 1) / best.tiles;
  if (best.G * best.tiles >= 2 * W) best.passes = kPhTile / (32 * F);
  return best;
}

// Models of more than kPqsLayers layers have a choice of kernels that give the same bits; how a
// block's time adds up decides it, and the split.  A step takes a warp `step` us by itself (latency)
// and the SM `pipe` us a warp once its warps fill the FP64 pipe; a layer of a slowness's prologue
// takes the SM `entry` us, and a round of the prologue's two stages 2.5 and 4 us (latency).
struct SweepKind {
  int nph, W, minb;
  double step, pipe, entry;
};
constexpr SweepKind kTableKind{2, 8, 2, 0.42, 0.056, 0.02};
constexpr SweepKind kLanesKind{kLanePhases, 4, 4, 0.55, 0.075, 0.01};
constexpr SweepKind kDirectKind4{0, 4, 4, 0.60, 0.085, 0.01};
constexpr SweepKind kDirectKind8{0, 8, 2, 0.60, 0.085, 0.01};

constexpr size_t kSmShared = 228 * 1024, kBlockShared = 1024 + sizeof(SweepTiles) + 64;

// The split of least estimated time, which it returns in *us.
static ForwardSplit forward_plan(long long n_p, int n_w, int L, const SweepKind& k, double* us) {
  const int n_wtiles = (n_w - 1) / kPhTile + 1, n_pass = (n_w - 1) / 32 + 1;
  ForwardSplit best{1, 1, n_wtiles, 1};
  *us = 1e300;
  for (int G = 1; G <= 16 && G <= n_p; ++G) {
    const size_t smem = sweep_block_bytes(L, k.nph, k.W, 1, G, n_pass) + kBlockShared;
    if (smem > kSmShared) break;
    const int resident = (int)(kSmShared / smem) < k.minb ? (int)(kSmShared / smem) : k.minb;
    for (int groups = 1; groups < 2 * n_wtiles; groups *= 2) {
      const int tiles = (n_wtiles + groups - 1) / groups;
      if (tiles > kSweepTiles) continue;
      const int passes = G * tiles >= 2 * k.W ? kPhTile / 32 : 1;
      const int tasks = passes > 1 ? G * tiles : G * (4 * tiles < n_pass ? 4 * tiles : n_pass);
      const int rounds = (tasks + k.W - 1) / k.W * passes, th = 32 * k.W;
      const int n_groups = (n_wtiles + tiles - 1) / tiles;
      const long long blocks = ((n_p + G - 1) / G) * n_groups;
      auto wave = [&](long long per_sm) {
        const double lat = rounds * k.step, pipe = (double)G * n_pass / n_groups * per_sm * k.pipe;
        return 2.5 * ((2 * G * L + th - 1) / th) + 4.0 * ((G * (L - 1) + th - 1) / th) +
               (L - 1) * (k.entry * G * per_sm + cbrt(lat * lat * lat + pipe * pipe * pipe));
      };
      const long long slots = 148LL * resident, rest = blocks % slots;
      const double t = (double)(blocks / slots) * wave(resident) +
                       (rest ? wave((rest + 147) / 148) : 0.0);
      if (t < 0.97 * *us) {
        *us = t;
        best = ForwardSplit{G, n_groups, tiles, passes};
      }
    }
  }
  return best;
}

template <class Form, int NPH, int F, int W, int MINB>
static kr_status launch_sweep_kernel(const char* what, const double* layers, int L, const double* p,
                                     int n_p, const double* omega, int n_w, uint32_t flags, double* R,
                                     cudaStream_t st, const ForwardSplit& s, size_t smem) {
  const int n_wtiles = (n_w - 1) / kPhTile + 1;
  const long long blocks = (((long long)n_p + s.G - 1) / s.G) * s.groups;
  if (blocks > 0x7fffffffLL) return KR_ERR_TOO_LARGE;
  static SmemLimit lim;
  if (smem > 46 * 1024) {  // with the static arrays above the 48 KB default
    const kr_status a = raise_smem_limit((const void*)sweep_kernel<Form, NPH, F, W, MINB>, smem,
                                         lim, what);
    if (a != KR_OK) return a;
  }
  sweep_kernel<Form, NPH, F, W, MINB><<<(unsigned)blocks, 32 * W, smem, st>>>(
      layers, L, p, n_p, reinterpret_cast<const double2*>(omega), n_w, n_wtiles, s.G, s.groups,
      s.tiles, s.passes, (flags & KR_FREE_SURFACE) ? 1 : 0, reinterpret_cast<double2*>(R));
  return check_launch(what);
}

// Models of up to kPqsLayers layers.
template <class Form, int NPH, int F, int W, int MINB>
static kr_status launch_forward(const char* what, const double* layers, int L, const double* p, int n_p,
                                const double* omega, int n_w, uint32_t flags, double* R,
                                cudaStream_t st) {
  const int n_wtiles = (n_w - 1) / kPhTile + 1;
  constexpr size_t kSm = 227 * 1024 - 8 * (sizeof(SweepTiles) + 16);
  const int n_pass = (n_w - 1) / (32 * F) + 1;
  const size_t one = sweep_block_bytes(L, NPH, W, F, 1, n_pass);
  int resident = (int)(kSm / (one + 1024));
  resident = resident < 1 ? 1 : resident > MINB ? MINB : resident;
  const ForwardSplit s =
      forward_split(n_p, n_wtiles, L, NPH, F, W, resident, kSm / resident - 1024, n_pass);
  return launch_sweep_kernel<Form, NPH, F, W, MINB>(what, layers, L, p, n_p, omega, n_w, flags, R, st,
                                                    s, sweep_block_bytes(L, NPH, W, F, s.G, n_pass));
}

// Deeper models: of the kernels that give the same bits the one with the least estimated time, a
// table or eight warps of direct exponentials where they do not clearly lose and win.  Microseconds
// with the table / by lanes: 513 x 31 of 48 layers 50 / 37, of 66 layers 64 / 50; 513 x 128 of 48
// layers 62 / 66; 2000 x 64 of 66 layers 257 / 184; 150 x 1024 of 66 layers 152 / 194.  With eight /
// four warps: 513 x 31 of 120 layers 98 / 82, 64 x 1024 of 120 layers 164 / 172, 150 x 300 of 120
// layers 188 / 171.  (One kernel for all of them, the table's or with eight warps, took 50, 87, 62,
// 287, 151, 148, 163 and 251.)
template <class Form>
static kr_status launch_forward_deep(const char* what, const double* layers, int L, const double* p,
                                     int n_p, const double* omega, int n_w, uint32_t flags, double* R,
                                     cudaStream_t st) {
  const bool pair = sweep_phases(L) == 2;
  const SweepKind& k0 = pair ? kTableKind : kDirectKind8;
  const SweepKind& k1 = pair ? kLanesKind : kDirectKind4;
  double t0, t1;
  const ForwardSplit s0 = forward_plan(n_p, n_w, L, k0, &t0);
  const ForwardSplit s1 = forward_plan(n_p, n_w, L, k1, &t1);
  const bool second = pair ? t1 < 0.95 * t0 : t1 <= 1.02 * t0;
  const ForwardSplit& s = second ? s1 : s0;
  const SweepKind& k = second ? k1 : k0;
  const size_t smem = sweep_block_bytes(L, k.nph, k.W, 1, s.G, (n_w - 1) / 32 + 1);
  if (pair)
    return second ? launch_sweep_kernel<Form, kLanePhases, 1, 4, 4>(what, layers, L, p, n_p, omega, n_w,
                                                                    flags, R, st, s, smem)
                  : launch_sweep_kernel<Form, 2, 1, 8, 2>(what, layers, L, p, n_p, omega, n_w, flags, R,
                                                          st, s, smem);
  return second ? launch_sweep_kernel<Form, 0, 1, 4, 4>(what, layers, L, p, n_p, omega, n_w, flags, R,
                                                        st, s, smem)
                : launch_sweep_kernel<Form, 0, 1, 8, 2>(what, layers, L, p, n_p, omega, n_w, flags, R, st,
                                                        s, smem);
}

}  // namespace kr
