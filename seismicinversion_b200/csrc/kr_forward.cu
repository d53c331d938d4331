// Fused forward reflectivity kernel: R[p][omega] of one model.
//
// A block takes G consecutive slownesses and a range of 128-frequency tiles.  Its prologue puts
// the layer terms, the interface coefficients and the phase tables of all G slownesses into
// shared memory; then its warps take tiles of 128 frequencies (or, where those are few, passes of
// 32 F) in turn, each running the whole bottom-up Kennett sweep with the cumulative reflection
// matrix in registers (kr_sweep.cuh), with no block barrier.  FP64 CUDA cores; no tensor-core
// work exists here (2x2 complex algebra per thread is not a contraction).
//
// The bound is the FP64 pipe fed by the register file: an FMA with three distinct register
// operands issues at 13.5e12 / s on this GPU (two operands: 18e12), and the 21-layer
// 8192 x 2047 grid runs at 12.9e12 (119 FP64 instructions per update, 3.1 ms; the form with
// two phases per step, a correctly rounded division and a block per slowness took 132 and
// 3.3 ms).  4096 x 2047 slownesses of a 5-layer model: 389 -> 322 us; 2048 x 511: 137 -> 58 us
// (several slownesses share a prologue); 193 x 1501 of a 64-layer model: 348 -> 253 us (table
// instead of direct exponentials).  Two frequencies per lane (half the coefficient loads, two
// chains) measured the same on 21 layers and 7 % slower on 5: registers, not loads, bound it.
#include <stdlib.h>

#include "kr_sweep.cuh"

namespace kr {

template <int NPH, int F, int W, int MINB>
__global__ void __launch_bounds__(32 * W, MINB)
reflectivity_kernel(const double* __restrict__ tab, int L, const double* __restrict__ p, int n_p,
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
  Iface* s_coef = reinterpret_cast<Iface*>(s_lay + (size_t)G * L);
  LayerRoots* s_root = reinterpret_cast<LayerRoots*>(s_coef + (size_t)G * I);
  cd* s_tab = reinterpret_cast<cd*>(s_root + (size_t)G * L);
  const int n_ent = NPH * I * kPhHead;  // table entries of one slowness
  cd* s_hm = s_tab + (size_t)G * n_ent;
  if (threadIdx.x == 0) s_bad = 0u;
  if (NPH > 0) sweep_tiles_clear(s_tiles, t1 - t0);
  for (int e = threadIdx.x; e < 2 * ng * L; e += 32 * W) {
    const int half = e >= ng * L ? 1 : 0, j = e - half * ng * L;
    layer_store(tab, L, j % L, half, p[ip0 + j / L], s_lay + j, s_root + j);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < ng * I; e += 32 * W) {
    const int g = e / I, i = e - g * I;
    interface_store(p[ip0 + g], i, s_lay + g * L, s_root + g * L, s_coef + e);
  }
  if (NPH > 0) {
    const GridLine line = grid_line(omega, n_w);
    sweep_tiles_check(omega, n_w, line, t0, t1 - t0, s_tiles);
    unsigned bad = 0u;
    for (int e = threadIdx.x; e < ng * n_ent; e += 32 * W) {
      const int g = e / n_ent, id = (e - g * n_ent) / kPhHead, j = e % kPhHead;
      if (!sweep_table_entry<N>(line, s_lay + g * L, id, j, s_tab + (size_t)g * n_ent))
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
    sweep_tile<NPH, F>(omega, NPH > 0 ? s_tiles.w0[v] : make_double2(0.0, 0.0), t0 + v, pass,
                       pass + passes, 0, n_w, L, s_lay + g * L, s_coef + g * I,
                       s_tab + (size_t)g * n_ent,
                       NPH > 0 && s_tiles.off[v] == 0 && ((bad >> g) & 1u) == 0u, hm,
                       free_surface != 0, R + (size_t)(ip0 + g) * n_w);
  }
}

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

template <int NPH, int F, int W, int MINB>
static kr_status launch_forward(const double* layers, int L, const double* p, int n_p,
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
    const kr_status a = raise_smem_limit((const void*)reflectivity_kernel<NPH, F, W, MINB>, smem,
                                         lim, "kr_reflectivity: smem attribute");
    if (a != KR_OK) return a;
  }
  reflectivity_kernel<NPH, F, W, MINB><<<(unsigned)blocks, 32 * W, smem, st>>>(
      layers, L, p, n_p, reinterpret_cast<const double2*>(omega), n_w, n_wtiles, s.G, s.groups,
      s.tiles, s.passes, (flags & KR_FREE_SURFACE) ? 1 : 0, reinterpret_cast<double2*>(R));
  return check_launch("kr_reflectivity");
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
  switch (sweep_phases(n_layers)) {
    case 0:
      return launch_forward<0, 1, 4, 4>(layers, n_layers, p, n_p, omega, n_w, flags, R, st);
    case 2:
      return launch_forward<2, 1, 8, 2>(layers, n_layers, p, n_p, omega, n_w, flags, R, st);
    default:
      switch (forward_minb()) {
        case 6:
          return launch_forward<3, 1, 4, 6>(layers, n_layers, p, n_p, omega, n_w, flags, R, st);
        case 5:
          return launch_forward<3, 1, 4, 5>(layers, n_layers, p, n_p, omega, n_w, flags, R, st);
        default:
          return launch_forward<3, 1, 4, 4>(layers, n_layers, p, n_p, omega, n_w, flags, R, st);
      }
  }
}
