// The forward sweep kernel and its launch, for any form of the recursion (kr_sweep.cuh).
//
// A block takes G consecutive slownesses and a range of 128-frequency tiles.  Its prologue puts
// the layer terms, the interface coefficients and the phase tables of all G slownesses into
// shared memory; then its warps take tiles of 128 frequencies (or, where those are few, passes of
// 32 F) in turn, each running the whole bottom-up sweep with the recursion's state in registers,
// with no block barrier.
#pragma once

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
  constexpr int N = NPH > 0 ? NPH : 1;
  const int I = L - 1;
  const int ip0 = (blockIdx.x / tile_groups) * G;
  const int ng = min(G, n_p - ip0);
  const int t0 = (blockIdx.x % tile_groups) * tiles_per_group;
  const int t1 = min(n_wtiles, t0 + tiles_per_group);
  LayerP* s_lay = reinterpret_cast<LayerP*>(smem);
  typedef typename Form::Coef Coef;
  static_assert(sizeof(Coef) <= sizeof(Iface), "sweep_slowness_bytes covers the form");
  Coef* s_coef = reinterpret_cast<Coef*>(s_lay + (size_t)G * L);
  LayerRoots* s_root = reinterpret_cast<LayerRoots*>(s_coef + (size_t)G * I);
  cd* s_tab = reinterpret_cast<cd*>(s_root + (size_t)G * L);
  const int n_ent = NPH * I * kPhHead;  // table entries of one slowness
  cd* s_hm = s_tab + (size_t)G * n_ent;
  if (threadIdx.x == 0) s_bad = 0u;
  for (int e = threadIdx.x; e < 2 * ng * L; e += 32 * W) {
    const int half = e >= ng * L ? 1 : 0, j = e - half * ng * L;
    layer_store(tab, L, j % L, half, p[ip0 + j / L], s_lay + j, s_root + j);
  }
  const GridLine line = grid_line(omega, n_w);
  bool on = NPH > 0 && sweep_tiles_check(omega, n_w, line, t0, t1 - t0, s_tiles);
  on = __syncthreads_or(on) != 0;
  for (int e = threadIdx.x; e < ng * I; e += 32 * W) {
    const int g = e / I, i = e - g * I;
    Form::store(p[ip0 + g], i, s_lay + g * L, s_root + g * L, s_coef + e);
  }
  if (NPH > 0 && on) {
    unsigned bad = 0u;
    for (int e = threadIdx.x; e < ng * I * kPhHead; e += 32 * W) {
      const int gl = e / kPhHead, g = gl / I;
      if (!sweep_table_entry<N>(line, s_lay + g * L, gl - g * I, e - gl * kPhHead,
                                s_tab + (size_t)g * n_ent))
        bad |= 1u << g;
    }
    if (bad) atomicOr(&s_bad, bad);
  }
  __syncthreads();
  const unsigned bad = s_bad;
  const int warp = threadIdx.x >> 5;
  cd* hm = s_hm + (size_t)warp * 2 * F * NPH * I;
  // tasks: (slowness, tile, `passes` of the tile's passes)
  const int parts = kPhTile / (32 * F) / passes;
  const int per_slowness = (t1 - t0) * parts;
  for (int t = warp; t < ng * per_slowness; t += W) {
    const int g = t / per_slowness, q = t - g * per_slowness;
    const int v = q / parts, pass = (q - v * parts) * passes;
    sweep_tile<Form, NPH, F>(omega, NPH > 0 ? s_tiles.w0[v] : make_double2(0.0, 0.0), t0 + v, pass,
                       pass + passes, 0, n_w, L, s_lay + g * L, s_coef + g * I,
                       s_tab + (size_t)g * n_ent,
                       NPH > 0 && s_tiles.off[v] == 0 && ((bad >> g) & 1u) == 0u, hm,
                       free_surface != 0, R + (size_t)(ip0 + g) * n_w);
  }
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
                                  int resident, size_t smem_max) {
  const size_t per = sweep_slowness_bytes(L, nph), fixed = W * sweep_warp_bytes(L, nph, F);
  ForwardSplit best{1, 1, n_wtiles, 1};
  double best_cost = 1e300;
  for (int G = 1; G <= 16; ++G) {
    if (G > 1 && (G * per + fixed > smem_max || G > n_p)) break;
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

template <class Form, int NPH, int F, int W, int MINB>
static kr_status launch_forward(const char* what, const double* layers, int L, const double* p, int n_p,
                                const double* omega, int n_w, uint32_t flags, double* R,
                                cudaStream_t st) {
  const int n_wtiles = (n_w + kPhTile - 1) / kPhTile;
  constexpr size_t kSm = 227 * 1024 - 8 * (sizeof(SweepTiles) + 16);
  const size_t fixed = W * sweep_warp_bytes(L, NPH, F);
  const size_t one = sweep_slowness_bytes(L, NPH) + fixed;
  int resident = (int)(kSm / (one + 1024));
  resident = resident < 1 ? 1 : resident > MINB ? MINB : resident;
  const ForwardSplit s =
      forward_split(n_p, n_wtiles, L, NPH, F, W, resident, kSm / resident - 1024);
  const size_t smem = s.G * sweep_slowness_bytes(L, NPH) + fixed;
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

}  // namespace kr
