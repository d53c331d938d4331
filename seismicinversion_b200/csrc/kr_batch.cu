// Batched evaluation of many earth models of uneven size in persistent launches.
//
// A batch is a list of models, each with its own layer count, slowness grid and frequency
// grid, asking for the forward reflectivity or forward + misfit gradient.  kr_batch_plan
// (host) builds, once per batch shape:
//   * a pair table: one entry per (model, slowness) with the offset of its coefficient block
//     in the plan buffer;
//   * two work lists (forward items, gradient items), item = (pair, first frequency, count),
//     models of more than 30 layers first, each class sorted by descending cost (layers x
//     frequencies, x4 for gradients) so the dynamic scheduler hands out the longest items
//     first (LPT);
// and uploads them into the caller's plan buffer.  kr_batch_launch (device only, capturable
// in a CUDA graph) then runs:
//   1. batch_prep_kernel: a group of threads per pair -> layer terms and interface coefficients
//      (and, for gradient models, layer derivative factors) into the plan;
//   2. batch_tan_kernel: the gradient models' coefficient tangents, one thread per interface
//      and tangent column, alongside the forward kernel (its programmatic dependent);
//   3. batch_forward_kernel (a launch for each depth class) and batch_grad_sums_kernel
//      (batch_gradient_kernel where a model's frequency sums exceed shared memory): persistent
//      grids (resident blocks only) that pull items with an atomic counter until the list is
//      exhausted.  Without observed data there are no gradient models and no launches for them.
// Gradient items reduce their contributions per block in a fixed order and add them to the
// model's chi_grad with FP64 atomics (the order of those additions across blocks is not
// fixed: results agree to rounding, ~1e-16 relative, run to run).
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "kr_adjoint.cuh"
#include "kr_adjsum.cuh"
#include "kr_internal.cuh"
#include "kr_sweep.cuh"

namespace kr {

struct PairRec {
  int32_t model;
  int32_t j;
  int64_t coef_off;  // bytes into the plan buffer
};

struct ItemRec {
  int32_t pair;
  int32_t w0;
  int32_t nw;
  int32_t pad;
};

struct PlanHeader {
  int32_t n_models, n_pairs, n_fwd, n_grad;
  int32_t threads, tile_w, grid_fwd, grid_grad;
  int64_t off_models, off_pairs, off_fwd, off_grad, total_bytes;
  int32_t n_fwd_deep, n_grad_deep;  // the lists' leading items, of models deeper than kPqsLayers
  int32_t counters[4];  // item counters: forward deep / shallow, gradient deep / shallow
};

__host__ __device__ inline size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

static size_t pair_bytes(const kr_model_desc& d) {
  const int L = d.n_layers, I = d.n_layers - 1;
  size_t b = a256(sizeof(LayerP) * L) + a256(sizeof(Iface) * I);
  if (d.flags & KR_BATCH_GRADIENT) b += a256(sizeof(LayerD) * L) + a256(sizeof(ScatTan) * I);
  return b;
}

struct PairView {
  const LayerP* lay;
  const Iface* coef;
  const LayerD* dlay;
  const ScatTan* tan;
};

__device__ __forceinline__ PairView pair_view(const unsigned char* plan, const PairRec& pr,
                                              const kr_model_desc& d) {
  const int L = d.n_layers, I = d.n_layers - 1;
  const unsigned char* b = plan + pr.coef_off;
  PairView v;
  v.lay = reinterpret_cast<const LayerP*>(b);
  b += a256(sizeof(LayerP) * L);
  v.coef = reinterpret_cast<const Iface*>(b);
  b += a256(sizeof(Iface) * I);
  v.dlay = reinterpret_cast<const LayerD*>(b);
  b += a256(sizeof(LayerD) * L);
  v.tan = reinterpret_cast<const ScatTan*>(b);
  return v;
}

// Layer terms, derivative factors (gradient models) and interface coefficients of every pair.
// A group of GS threads takes a pair: GS is the power of two that covers the deepest model's
// layers (4 to 64), so a batch of 5-layer models keeps all of a warp's lanes busy (eight
// threads a pair) where a block a pair left 59 of 64 threads idle (49152 pairs of 5 layers:
// 360 us).  A pair's threads meet at a warp or (GS = 64) block barrier between the layer terms
// and the coefficients that read them back; every group of a block runs the same number of
// rounds.
constexpr int kPrepBlock = 64;

__global__ void __launch_bounds__(kPrepBlock)
batch_prep_kernel(unsigned char* plan, const double* __restrict__ layers,
                  const double* __restrict__ p_all, int gs) {
  __shared__ LayerRoots s_roots[kMaxLayers];  // kMaxLayers / groups per group, at least gs
  const PlanHeader* h = reinterpret_cast<const PlanHeader*>(plan);
  const kr_model_desc* models = reinterpret_cast<const kr_model_desc*>(plan + h->off_models);
  const PairRec* pairs = reinterpret_cast<const PairRec*>(plan + h->off_pairs);
  const int groups = kPrepBlock / gs, mine = threadIdx.x / gs, t0 = threadIdx.x % gs;
  const int stride = gridDim.x * groups;
  for (int q0 = blockIdx.x * groups; q0 < h->n_pairs; q0 += stride) {
    const int q = q0 + mine;
    const bool have = q < h->n_pairs;
    const PairRec pr = pairs[have ? q : q0];
    const kr_model_desc d = models[pr.model];
    const int L = have ? d.n_layers : 0, I = L - 1;
    const double* tab = layers + d.layers_off;
    const double pj = p_all[d.p_off + pr.j];
    unsigned char* b = plan + pr.coef_off;
    LayerP* lay = reinterpret_cast<LayerP*>(b);
    b += a256(sizeof(LayerP) * d.n_layers);
    Iface* coef = reinterpret_cast<Iface*>(b);
    b += a256(sizeof(Iface) * (d.n_layers - 1));
    LayerD* dlay = reinterpret_cast<LayerD*>(b);
    const bool grad = (d.flags & KR_BATCH_GRADIENT) != 0;
    LayerRoots* roots = s_roots + mine * (kMaxLayers / kPrepBlock) * gs;
    for (int t = t0; t < 2 * L; t += gs) {
      const int half = t >= L ? 1 : 0, l = t - half * L;
      layer_store(tab, L, l, half, pj, lay + l, roots + l);
    }
    if (gs > 32) __syncthreads(); else __syncwarp();
    for (int i = t0; i < I; i += gs) interface_store(pj, i, lay, roots + i, roots + i + 1, coef + i);
    if (grad)
      for (int l = t0; l < L; l += gs) dlay[l] = layer_derivs(tab, L, l, pj, lay[l]);
    if (gs > 32) __syncthreads(); else __syncwarp();  // the roots are read before the next pair's
  }
}

// Coefficient tangents of the gradient models' pairs, one thread per (interface, tangent
// column), from the layer terms and derivative factors batch_prep_kernel left in the plan.
// Only the gradient kernel reads them, so the forward kernel is launched as this kernel's
// programmatic dependent (released on entry) and runs alongside it; the forward kernel
// waits for this grid before it exits, so the gradient kernel after it sees the tangents.
__global__ void __launch_bounds__(64)
batch_tan_kernel(unsigned char* plan, const double* __restrict__ p_all) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const PlanHeader* h = reinterpret_cast<const PlanHeader*>(plan);
  const kr_model_desc* models = reinterpret_cast<const kr_model_desc*>(plan + h->off_models);
  const PairRec* pairs = reinterpret_cast<const PairRec*>(plan + h->off_pairs);
  for (int q = blockIdx.x; q < h->n_pairs; q += gridDim.x) {
    const PairRec pr = pairs[q];
    const kr_model_desc d = models[pr.model];
    if (!(d.flags & KR_BATCH_GRADIENT)) continue;
    const int L = d.n_layers, I = L - 1;
    const double pj = p_all[d.p_off + pr.j];
    unsigned char* b = plan + pr.coef_off;
    const LayerP* lay = reinterpret_cast<const LayerP*>(b);
    b += a256(sizeof(LayerP) * L) + a256(sizeof(Iface) * I);
    const LayerD* dlay = reinterpret_cast<const LayerD*>(b);
    b += a256(sizeof(LayerD) * L);
    ScatTan* tan = reinterpret_cast<ScatTan*>(b);
    for (int t = threadIdx.x; t < 6 * I; t += blockDim.x) {
      const int i = t / 6, col = t % 6;
      cd c[10];
      interface_tangent_col(pj, i, lay[i], dlay[i], lay[i + 1], dlay[i + 1], col, c);
      for (int k = 0; k < 10; ++k) tan[i].t[k][col] = c[k];
    }
  }
}

// Zeroes chi_grad of gradient models and the item counters (first node of a launch).
__global__ void batch_reset_kernel(unsigned char* plan, double* chi_grad) {
  PlanHeader* h = reinterpret_cast<PlanHeader*>(plan);
  const kr_model_desc* models = reinterpret_cast<const kr_model_desc*>(plan + h->off_models);
  if (blockIdx.x == 0 && threadIdx.x < 4) h->counters[threadIdx.x] = 0;
  for (int b = blockIdx.x; b < h->n_models; b += gridDim.x) {
    const kr_model_desc d = models[b];
    if (!(d.flags & KR_BATCH_GRADIENT)) continue;
    for (int k = threadIdx.x; k < 4 * d.n_layers + 1; k += blockDim.x) chi_grad[d.grad_off + k] = 0.0;
  }
}

// The block's work items from a shared counter.  The next item's number is fetched while the
// current one is processed, so the atomic's latency does not sit between short items.
struct ItemFeed {
  int* counter;
  int* slot;  // one shared word
  int ahead;  // thread 0: the number fetched ahead
  __device__ __forceinline__ ItemFeed(int* c, int* s) : counter(c), slot(s), ahead(0) {
    if (threadIdx.x == 0) ahead = atomicAdd(counter, 1);
  }
  // Contains block barriers: every thread is done with the previous item.
  __device__ __forceinline__ int next() {
    __syncthreads();
    if (threadIdx.x == 0) {
      *slot = ahead;
      ahead = atomicAdd(counter, 1);
    }
    __syncthreads();
    return *slot;
  }
};

// Forward items: one (model, slowness) pair and a frequency range [w0, w0 + nw).  The block
// copies the pair's layer terms and coefficients from the plan, builds its phase table and its
// warps take the passes of the range in turn (kr_sweep.cuh: the code of kr_reflectivity, so the
// results are bit-identical to a per-model call).  CLASS selects the class of the work list:
// models of up to kPqsLayers layers, whose blocks are small, or deeper ones; each class is one
// persistent launch with the shared memory and registers of its own models, so that a batch's
// shallow models do not run at the occupancy of its deepest.  The deep class has two kernels that give
// the same bits: with phase tables (98 KB for 66 layers and 128 threads, two blocks per SM) and with
// phases formed by the lanes (45 KB, four), which direct exponentials beyond 66 layers share.  Items
// of one or two passes, and batches with models beyond 66 layers, take the second: 500 x 12 x 64 of
// 48 layers 531 us with tables, 395 without; 64 x 12 x 31 of 80 layers 184 with the tables' two blocks
// per SM, 144 without; 96 uneven models of up to 64 layers 10.70 ms with tables, 11.32 without.
enum ForwardClass { kShallow, kDeepTable, kDeepLanes };

template <int NPH, int F, int THREADS>
__device__ __forceinline__ void forward_item(const ItemRec& item, const kr_model_desc& d, int j,
                                             const PairView& v, const double2* om, double2* Rp,
                                             unsigned char* smem, SweepTiles& tiles) {
  constexpr bool kTable = NPH > 1, kLanes = NPH == kLanePhases;
  constexpr int N = kTable ? NPH : 2;
  const int L = d.n_layers, I = L - 1;
  LayerP* lay = reinterpret_cast<LayerP*>(smem);
  Iface* coef = reinterpret_cast<Iface*>(lay + L);
  cd* tab = reinterpret_cast<cd*>(coef + I);
  cd* hm = tab + (kTable ? (size_t)NPH * I * kPhHead : 0) +
           (size_t)(threadIdx.x >> 5) * 2 * F * (kLanes ? 2 : NPH) * I;
  const int u0 = item.w0 / kPhTile, n_tiles = (item.w0 + item.nw - 1) / kPhTile - u0 + 1;
  copy16(lay, v.lay, sizeof(LayerP) * L);
  copy16(coef, v.coef, sizeof(Iface) * I);
  const GridLine g = grid_line(om, d.n_w);
  bool on = NPH > 0 && sweep_tiles_check(om, d.n_w, g, u0, n_tiles, tiles);
  on = __syncthreads_or(on) != 0;
  bool bad = false;
  if (kLanes && on)
    for (int e = threadIdx.x; e < 2 * I; e += THREADS) bad |= !phase_table_usable(g, sweep_exponent(lay, e));
  if (kTable && on) {
    // an item within one tile needs only the mid entries of its own frequencies
    const int m0 = n_tiles > 1 ? 0 : (item.w0 % kPhTile) / kPhLo;
    const int m1 = n_tiles > 1 ? kPhMid : ((item.w0 + item.nw - 1) % kPhTile) / kPhLo + 1;
    const int per = kPhLo + m1 - m0;
    for (int e = threadIdx.x; e < I * per; e += THREADS) {
      const int l = e / per, j = e - l * per;
      bad |= !sweep_table_entry<N>(g, lay, l, j < kPhLo ? j : j + m0, tab);
    }
  }
  const bool ok = __syncthreads_or(bad) == 0;
  constexpr int kPasses = kPhTile / (32 * F);
  // a warp takes whole tiles, or single passes of short items
  const int passes = n_tiles >= 2 * (THREADS / 32) ? kPasses : 1, parts = kPasses / passes;
  for (int t = threadIdx.x >> 5; t < n_tiles * parts; t += THREADS / 32) {
    const int q = t / parts, pass = (t - q * parts) * passes;
    const double2 w0 = NPH > 0 ? tiles.w0[q] : make_double2(0.0, 0.0);
    const bool use = NPH > 0 && ok && tiles.off[q] == 0, fs = (d.flags & KR_FREE_SURFACE) != 0;
    if (kLanes)
      sweep_tile_lanes<KennettForm>(om, g, w0, u0 + q, pass, pass + passes, item.w0, item.w0 + item.nw,
                                    L, lay, coef, use, hm, fs, Rp);
    else
      sweep_tile<KennettForm, kTable ? NPH : 0, F>(om, w0, u0 + q, pass, pass + passes, item.w0,
                                                   item.w0 + item.nw, L, lay, coef, tab, use, hm, fs, Rp);
  }
}

template <int THREADS, ForwardClass CLASS>
__global__ void __launch_bounds__(THREADS, (CLASS == kDeepTable ? 256 : 512) / THREADS)
batch_forward_kernel(unsigned char* plan, const double2* __restrict__ omega_all,
                     double2* __restrict__ R_all) {
  // the next launch on the stream that allows it may fill in as this one's blocks finish
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr bool DEEP = CLASS != kShallow;
  extern __shared__ __align__(16) unsigned char s_pair[];
  __shared__ SweepTiles s_tiles;
  PlanHeader* h = reinterpret_cast<PlanHeader*>(plan);
  const kr_model_desc* models = reinterpret_cast<const kr_model_desc*>(plan + h->off_models);
  const PairRec* pairs = reinterpret_cast<const PairRec*>(plan + h->off_pairs);
  const ItemRec* items = reinterpret_cast<const ItemRec*>(plan + h->off_fwd) +
                         (DEEP ? 0 : h->n_fwd_deep);
  const int n_items = DEEP ? h->n_fwd_deep : h->n_fwd - h->n_fwd_deep;
  __shared__ int s_item;
  ItemFeed feed(&h->counters[DEEP ? 0 : 1], &s_item);
  for (;;) {
    const int it = feed.next();
    if (it >= n_items) break;
    const ItemRec item = items[it];
    const PairRec pr = pairs[item.pair];
    const kr_model_desc d = models[pr.model];
    const PairView v = pair_view(plan, pr, d);
    const double2* om = omega_all + d.omega_off;
    double2* Rp = R_all + d.R_off + (size_t)pr.j * d.n_w;
    if (!DEEP)
      forward_item<3, 1, THREADS>(item, d, pr.j, v, om, Rp, s_pair, s_tiles);
    else if (CLASS == kDeepTable)
      forward_item<2, 1, THREADS>(item, d, pr.j, v, om, Rp, s_pair, s_tiles);
    else if (sweep_phases(d.n_layers) == 2)
      forward_item<kLanePhases, 1, THREADS>(item, d, pr.j, v, om, Rp, s_pair, s_tiles);
    else
      forward_item<0, 1, THREADS>(item, d, pr.j, v, om, Rp, s_pair, s_tiles);
  }
  // launched as its predecessor's programmatic dependent: this grid completes only after that
  // one has, so the gradient kernel launched after it reads finished tangents
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Per-thread sink for gradient items: 2 Re(conj(res) dR/dtheta) per layer, reduced over the
// warp by shuffles into the warp's own accumulator row (no block barrier inside the sweep).
template <int THREADS>
struct BatchGradSink {
  typedef AccR AccT;  // reverse sweep seeded with 2 conj(res): real contributions only
  static constexpr bool kSeeded = true;
  bool valid;
  cd res;
  const double2* obs;
  double2* R_out;
  double* row;  // this warp's [4L + 1] accumulators
  int L;
  __device__ cd reflectivity(cd R) {
    res = mk(0.0, 0.0);
    if (!valid) return mk(0.0, 0.0);
    if (R_out) *R_out = make_double2(R.x, R.y);
    const double2 o = *obs;
    res = mk(R.x - o.x, R.y - o.y);
    return mk(2.0 * res.x, -2.0 * res.y);  // 2 conj(res)
  }
  __device__ void layer(int l, const AccR& a) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (valid) {
      v[0] = a.a;
      v[1] = a.b;
      v[2] = a.r;
      v[3] = a.h;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0)
      for (int k = 0; k < 4; ++k) row[k * L + l] += v[k];
  }
};

// Passes of 32 frequencies of an item: the warp's first pass and its stride are in units of whole
// warps, so that every pass lies in one tile and its phases come from two hm entries.
#define KR_FOR_PASSES(kb) \
  for (int kb = (item.w0 & ~31) + (int)(threadIdx.x & ~31u); kb < item.w0 + item.nw; kb += THREADS)

// The tile verdicts and (models that tabulate) lo entries of a gradient item; returns whether its
// tiles on the line take the table, or PhaseLine.  `lay` may still be on its way from other threads:
// contains block barriers; all threads call it.
__device__ __forceinline__ bool ray_item_tables(const ItemRec& item, const kr_model_desc& d,
                                                const double2* om, const LayerP* lay, cd* lo,
                                                SweepTiles& tiles) {
  const int u0 = item.w0 / kPhTile, n = (item.w0 + item.nw - 1) / kPhTile - u0 + 1;
  const GridLine g = grid_line(om, d.n_w);
  bool on = ray_line_model(d.n_layers) && sweep_tiles_check(om, d.n_w, g, u0, n, tiles);
  on = __syncthreads_or(on) != 0;
  if (!on || !ray_table_model(d.n_layers)) return on;
  return __syncthreads_and(ray_lo_fill(g, d.n_layers, lay, lo)) != 0;
}

// Gradient items of models whose frequency sums exceed shared memory (more than ~118 layers in
// the batch; all of them with KR_DERIV_SUMS=0): the contraction per (omega, p), as
// deriv_sweep_kernel.  `deep`: the class of the work list.
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
batch_gradient_kernel(unsigned char* plan, const double2* __restrict__ omega_all,
                      const double2* __restrict__ obs_all, double2* __restrict__ R_all,
                      double* __restrict__ chi_grad, int stage, int deep) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // [THREADS / 32][4L + 1] accumulators (padded to 16 bytes), then (models that tabulate) the
  // phase table, then, if `stage`, the item's slowness data
  extern __shared__ __align__(16) double s_wacc[];
  __shared__ SweepTiles s_tiles;
  PlanHeader* h = reinterpret_cast<PlanHeader*>(plan);
  const kr_model_desc* models = reinterpret_cast<const kr_model_desc*>(plan + h->off_models);
  const PairRec* pairs = reinterpret_cast<const PairRec*>(plan + h->off_pairs);
  const ItemRec* items = reinterpret_cast<const ItemRec*>(plan + h->off_grad) +
                         (deep ? 0 : h->n_grad_deep);
  const int n_items = deep ? h->n_grad_deep : h->n_grad - h->n_grad_deep;
  __shared__ int s_item;
  ItemFeed feed(&h->counters[deep ? 2 : 3], &s_item);
  for (;;) {
    const int it = feed.next();
    if (it >= n_items) break;
    const ItemRec item = items[it];
    const PairRec pr = pairs[item.pair];
    const kr_model_desc d = models[pr.model];
    PairView v = pair_view(plan, pr, d);
    const int L = d.n_layers;
    const int nv = 4 * L + 1;
    for (int k = threadIdx.x; k < (THREADS / 32) * nv; k += THREADS) s_wacc[k] = 0.0;
    cd* lo = reinterpret_cast<cd*>(s_wacc + ((THREADS / 32) * nv + 1) / 2 * 2);
    unsigned char* b = reinterpret_cast<unsigned char*>(lo);
    if (ray_table_model(L)) b += ray_table_bytes(L, THREADS / 32);
    if (stage) {
      ScatTan* st = reinterpret_cast<ScatTan*>(b);
      Iface* sc = reinterpret_cast<Iface*>(b + sizeof(ScatTan) * (L - 1));
      LayerP* sl = reinterpret_cast<LayerP*>(b + (sizeof(ScatTan) + sizeof(Iface)) * (L - 1));
      LayerD* sd = reinterpret_cast<LayerD*>(reinterpret_cast<unsigned char*>(sl) +
                                             sizeof(LayerP) * L);
      copy16(st, v.tan, sizeof(ScatTan) * (L - 1));
      copy16(sc, v.coef, sizeof(Iface) * (L - 1));
      copy16(sl, v.lay, sizeof(LayerP) * L);
      copy16(sd, v.dlay, sizeof(LayerD) * L);
      v.tan = st;
      v.coef = sc;
      v.lay = sl;
      v.dlay = sd;
    }
    const double2* om = omega_all + d.omega_off;
    const bool lo_ok = ray_item_tables(item, d, om, v.lay, lo, s_tiles);
    cd* hm = lo + ray_lo_values(L) + (threadIdx.x >> 5) * ray_hm_values(L);
    double* row = s_wacc + (threadIdx.x >> 5) * nv;
    const int seg = checkpoint_spacing(L - 2 > 0 ? L - 2 : 1);
    const bool fs = (d.flags & KR_FREE_SURFACE) != 0;
    KR_FOR_PASSES(kb) {
      const int iw = kb + (threadIdx.x & 31);
      const bool valid = iw >= item.w0 && iw < item.w0 + item.nw;
      const double2 wv = om[min(iw, d.n_w - 1)];
      const cd w = mk(wv.x, wv.y);
      BatchGradSink<THREADS> sink;
      sink.valid = valid;
      sink.L = L;
      sink.row = row;
      const size_t e = (size_t)pr.j * d.n_w + (valid ? iw : 0);
      sink.obs = obs_all + d.obs_off + e;
      sink.R_out = (d.flags & KR_BATCH_STORE_R) ? R_all + d.R_off + e : nullptr;
      const bool on = lo_ok && s_tiles.off[kb / kPhTile - item.w0 / kPhTile] == 0;
      const bool grow = warp_grows(valid, w);
      const bool tab =
          on && !grow && ray_table_model(L) && ray_hm_fill(om, d.n_w, kb, L, v.lay, hm);
      if (tab)
        jacobian_pair(L, w, fs, seg, v.lay, v.dlay, v.coef, v.tan, ray_table(lo, hm), sink);
      else
        jacobian_pair(L, w, fs, seg, v.lay, v.dlay, v.coef, v.tan,
                      PhaseEither(phase_line(on && (grow || !ray_table_model(L)), om, d.n_w, iw, w,
                                             v.lay), grow), sink);
      __syncwarp();
      double c2 = valid ? (sink.res.x * sink.res.x + sink.res.y * sink.res.y) : 0.0;
      for (int o = 16; o > 0; o >>= 1) c2 += __shfl_down_sync(0xffffffffu, c2, o);
      if ((threadIdx.x & 31) == 0) row[4 * L] += c2;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nv; k += THREADS) {
      double t = 0.0;
      for (int wi = 0; wi < THREADS / 32; ++wi) t += s_wacc[wi * nv + k];
      atomicAdd(chi_grad + d.grad_off + k, t);
    }
  }
}

// Gradient items with the contraction moved out of the frequency loop (kr_adjsum.cuh): the
// block's warps take the item's passes of 32 frequencies in turn and sum the per-step adjoints
// into their rows; the block contracts once per (pair, interface).  Dynamic smem, laid out for
// the item's own model: per-warp sum rows and staging rows (which then hold the item's [4L]
// result), interface coefficients and layer terms, and (models that tabulate) the phase table.
// Two depth classes as in the forward kernel: three blocks of 128 threads per SM for models of
// up to 30 layers (72 KB), two for deeper ones (107 KB).
template <int THREADS, bool DEEP>
__global__ void __launch_bounds__(THREADS, (DEEP ? 256 : 384) / THREADS)
batch_grad_sums_kernel(unsigned char* plan, const double2* __restrict__ omega_all,
                       const double2* __restrict__ obs_all, double2* __restrict__ R_all,
                       double* __restrict__ chi_grad) {
  // the other class may fill in as this one's blocks finish
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int W = THREADS / 32;
  extern __shared__ __align__(16) double s_raw[];
  __shared__ SweepTiles s_tiles;
  __shared__ double s_chi[W];
  PlanHeader* h = reinterpret_cast<PlanHeader*>(plan);
  const kr_model_desc* models = reinterpret_cast<const kr_model_desc*>(plan + h->off_models);
  const PairRec* pairs = reinterpret_cast<const PairRec*>(plan + h->off_pairs);
  const ItemRec* items = reinterpret_cast<const ItemRec*>(plan + h->off_grad) +
                         (DEEP ? 0 : h->n_grad_deep);
  const int n_items = DEEP ? h->n_grad_deep : h->n_grad - h->n_grad_deep;
  const int warp = threadIdx.x >> 5;
  __shared__ int s_item;
  ItemFeed feed(&h->counters[DEEP ? 2 : 3], &s_item);
  for (;;) {
    const int it = feed.next();
    if (it >= n_items) break;
    const ItemRec item = items[it];
    const PairRec pr = pairs[item.pair];
    const kr_model_desc d = models[pr.model];
    const PairView v = pair_view(plan, pr, d);
    const int L = d.n_layers, I = L - 1;
    double* acc = s_raw;
    cd* stage = reinterpret_cast<cd*>(acc + (size_t)W * sum_rows(L) * kRayRow);
    Iface* sc = reinterpret_cast<Iface*>(stage + W * kRayStage);
    LayerP* sl = reinterpret_cast<LayerP*>(sc + I);
    cd* lo = reinterpret_cast<cd*>(sl + L);
    cd* hm = lo + ray_lo_values(L) + warp * ray_hm_values(L);
    sums_zero(acc, L, W);
    copy16(sc, v.coef, sizeof(Iface) * I);
    copy16(sl, v.lay, sizeof(LayerP) * L);
    const double2* om = omega_all + d.omega_off;
    const bool lo_ok = ray_item_tables(item, d, om, sl, lo, s_tiles);
    const int seg = checkpoint_spacing(L - 2 > 0 ? L - 2 : 1);
    const bool fs = (d.flags & KR_FREE_SURFACE) != 0;
    double c2 = 0.0;
    KR_FOR_PASSES(kb) {
      const int iw = kb + (threadIdx.x & 31);
      const bool valid = iw >= item.w0 && iw < item.w0 + item.nw;
      const double2 wv = om[min(iw, d.n_w - 1)];
      const cd w = mk(wv.x, wv.y);
      const size_t e = (size_t)pr.j * d.n_w + (valid ? iw : 0);
      RaySumSink sink;
      sink.valid = valid;
      sink.vjp = false;
      sink.obs = obs_all + d.obs_off + e;
      sink.R_out = (d.flags & KR_BATCH_STORE_R) ? R_all + d.R_off + e : nullptr;
      sink.acc = acc + (size_t)warp * sum_rows(L) * kRayRow;
      sink.stage = stage + warp * kRayStage;
      sink.I = I;
      const bool on = lo_ok && s_tiles.off[kb / kPhTile - item.w0 / kPhTile] == 0;
      const bool grow = warp_grows(valid, w);
      const bool tab =
          on && !grow && ray_table_model(L) && ray_hm_fill(om, d.n_w, kb, L, sl, hm);
      if (tab)
        adjoint_rays(L, w, fs, seg, sc, ray_table(lo, hm), sink);
      else if (!grow)
        adjoint_rays(L, w, fs, seg, sc,
                     phase_line(on && !ray_table_model(L), om, d.n_w, iw, w, sl), sink);
      else
        adjoint_rays(L, w, fs, seg, sc, PhaseGrown(phase_line(on, om, d.n_w, iw, w, sl)), sink);
      __syncwarp();  // the hm entries are read before the next pass overwrites them
      if (valid) c2 += sink.res.x * sink.res.x + sink.res.y * sink.res.y;
    }
    for (int o = 16; o > 0; o >>= 1) c2 += __shfl_down_sync(0xffffffffu, c2, o);
    if ((threadIdx.x & 31) == 0) s_chi[warp] = c2;
    // the item's [4L] result goes where the staging rows were
    double* s_out = reinterpret_cast<double*>(stage);
    sums_finish(acc, L, W, v.tan, v.dlay, s_out);
    __syncthreads();
    for (int k = threadIdx.x; k < 4 * L; k += THREADS) atomicAdd(chi_grad + d.grad_off + k, s_out[k]);
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int wi = 0; wi < W; ++wi) t += s_chi[wi];
      atomicAdd(chi_grad + d.grad_off + 4 * L, t);
    }
  }
  // complete only after the class launched before this one
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

static int occupancy_grid(const void* fn, int threads, size_t smem) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return per_sm * sms;
}

static bool valid_config(const kr_batch_config* c) {
  return c && (c->threads == 32 || c->threads == 64 || c->threads == 128) && c->tile_w >= 32 &&
         c->tile_w <= 8192;
}

// The layout of a plan needs counts only; the lists themselves are written by plan_image.
struct PlanLayout {
  PlanHeader h;
  int64_t off_coef;  // the first pair's coefficient block (and the metadata's end, aligned)
  size_t bytes;
};

static kr_status layout(const kr_model_desc* descs, int n_models, const kr_batch_config* cfg,
                        PlanLayout* out) {
  PlanHeader h{};
  h.n_models = n_models;
  h.threads = cfg->threads;
  h.tile_w = cfg->tile_w;
  long long n_pairs = 0, n_fwd = 0, n_grad = 0, n_fwd_deep = 0, n_grad_deep = 0;
  size_t coef = 0;
  for (int b = 0; b < n_models; ++b) {
    const kr_model_desc& d = descs[b];
    if (d.n_layers < 2) return KR_ERR_INVALID_MODEL;
    if (d.n_layers > kMaxLayers) return KR_ERR_TOO_LARGE;
    if (d.n_p < 0 || d.n_w < 0 || (d.flags & ~(KR_FREE_SURFACE | KR_BATCH_GRADIENT |
                                               KR_BATCH_STORE_R)))
      return KR_ERR_INVALID_ARGUMENT;
    const bool gr = (d.flags & KR_BATCH_GRADIENT) != 0;
    n_pairs += d.n_p;
    const long long items = (long long)d.n_p * ((d.n_w + cfg->tile_w - 1) / cfg->tile_w);
    (gr ? n_grad : n_fwd) += items;
    if (d.n_layers > kPqsLayers) (gr ? n_grad_deep : n_fwd_deep) += items;
    coef += pair_bytes(d) * (size_t)d.n_p;
  }
  if (n_pairs > 0x7fffffffLL || n_fwd > 0x7fffffffLL || n_grad > 0x7fffffffLL)
    return KR_ERR_TOO_LARGE;
  h.n_pairs = (int)n_pairs;
  h.n_fwd = (int)n_fwd;
  h.n_grad = (int)n_grad;
  h.n_fwd_deep = (int)n_fwd_deep;
  h.n_grad_deep = (int)n_grad_deep;
  size_t off = a256(sizeof(PlanHeader));
  h.off_models = (int64_t)off;
  off = a256(off + sizeof(kr_model_desc) * (size_t)n_models);
  h.off_pairs = (int64_t)off;
  off = a256(off + sizeof(PairRec) * (size_t)n_pairs);
  h.off_fwd = (int64_t)off;
  off = a256(off + sizeof(ItemRec) * (size_t)n_fwd);
  h.off_grad = (int64_t)off;
  off = a256(off + sizeof(ItemRec) * (size_t)n_grad);
  out->off_coef = (int64_t)off;
  h.total_bytes = (int64_t)(off + coef);
  out->h = h;
  out->bytes = off + coef;
  return KR_OK;
}

constexpr size_t kBatchStageMax = 160 * 1024;

// Shared memory of a class of the forward kernel for models of up to max_layers.
static size_t fwd_smem(int threads, int max_layers, ForwardClass c) {
  const int w = threads / 32, L = std::min(max_layers, c == kShallow ? kPqsLayers : kPairLayers);
  if (c != kDeepLanes) {
    const int nph = c == kShallow ? 3 : 2;
    return sweep_slowness_bytes(L, nph) + w * sweep_warp_bytes(L, nph, 1);
  }
  return std::max(prologue_smem_bytes(L) + w * sweep_warp_bytes(L, kLanePhases, 1),
                  prologue_smem_bytes(max_layers));
}

// batch_gradient_kernel's dynamic smem and whether the slowness data is staged.
static size_t grad_smem(int threads, int max_layers, int* stage) {
  const size_t acc = sizeof(double) * (((size_t)(threads / 32) * (4 * max_layers + 1) + 1) / 2 * 2);
  const size_t table = ray_table_bytes(std::min(max_layers, kRayTabLayers), threads / 32);
  const size_t pair = pair_smem_bytes(max_layers);
  *stage = (acc + table + pair <= kBatchStageMax) ? 1 : 0;
  return acc + table + (*stage ? pair : 0);
}

// Dynamic smem of batch_grad_sums_kernel for models of up to max_layers (0 if it does not fit):
// the largest of its models, which need not be the deepest, as only some tabulate.
static size_t sums_smem(int threads, int max_layers) {
  const int w = threads / 32;
  size_t most = 0;
  for (int L = 2; L <= max_layers; ++L) {
    const size_t b = raysum_smem_bytes(L, w) + prologue_smem_bytes(L) +
                     (ray_table_model(L) ? ray_table_bytes(L, w) : 0);
    most = std::max(most, b);
  }
  // the staging rows hold the item's [4L] result after its sweeps
  if (sizeof(cd) * kRayStage * (threads / 32) < sizeof(double) * 4 * (size_t)max_layers) return 0;
  return most <= kBatchStageMax ? most : 0;
}

// KR_DERIV_SUMS=0 keeps the per-step contraction for gradient items (comparison runs).
static bool batch_sums_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("KR_DERIV_SUMS");
    v = (e && atoi(e) == 0) ? 0 : 1;
  }
  return v == 1;
}

}  // namespace kr

using namespace kr;

extern "C" size_t kr_batch_plan_bytes(const kr_model_desc* descs, int32_t n_models,
                                      const kr_batch_config* cfg) {
  if (!descs || n_models < 0 || !valid_config(cfg)) return 0;
  PlanLayout lay;
  if (layout(descs, n_models, cfg, &lay) != KR_OK) return 0;
  return lay.bytes;
}

static size_t meta_bytes(const PlanLayout& lay) {
  return (size_t)lay.h.off_grad + sizeof(ItemRec) * (size_t)lay.h.n_grad;
}

// Fills the plan's metadata image (header, model table, pair table, work lists) of
// meta_bytes(lay) bytes.  Host only: no CUDA call.  Items of one model differ in cost only
// between its full frequency ranges and its last, shorter one, so the lists are sorted as
// groups (model, full or last range), deep models first, by descending cost and then written out: planning 4096
// models of 12 slownesses took four passes of 1.4 to 3.9 ms, two of them sorting 49152 items.
static void plan_image(const kr_model_desc* descs, int n_models, const kr_batch_config* cfg,
                       const PlanLayout& lay, unsigned char* img) {
  memset(img, 0, meta_bytes(lay));
  memcpy(img, &lay.h, sizeof(PlanHeader));
  memcpy(img + lay.h.off_models, descs, sizeof(kr_model_desc) * (size_t)n_models);
  PairRec* pairs = reinterpret_cast<PairRec*>(img + lay.h.off_pairs);
  struct Group {
    double cost;
    int model, first_pair;
    bool last;  // the model's last, shorter frequency range
  };
  std::vector<Group> fwd, grad;
  int64_t off = lay.off_coef;
  int q = 0;
  for (int b = 0; b < n_models; ++b) {
    const kr_model_desc& d = descs[b];
    const int64_t pb = (int64_t)pair_bytes(d);
    const bool gr = (d.flags & KR_BATCH_GRADIENT) != 0;
    const double unit = (double)(d.n_layers - 1) * (gr ? 4.0 : 1.0);
    std::vector<Group>& list = gr ? grad : fwd;
    if (d.n_p > 0) {
      if (d.n_w >= cfg->tile_w) list.push_back(Group{unit * cfg->tile_w, b, q, false});
      if (d.n_w % cfg->tile_w) list.push_back(Group{unit * (d.n_w % cfg->tile_w), b, q, true});
    }
    for (int j = 0; j < d.n_p; ++j, ++q, off += pb) pairs[q] = PairRec{b, j, off};
  }
  auto write = [&](std::vector<Group>& list, ItemRec* it) {
    std::stable_sort(list.begin(), list.end(), [&](const Group& a, const Group& b) {
      const bool da = descs[a.model].n_layers > kPqsLayers;
      const bool db = descs[b.model].n_layers > kPqsLayers;
      return da != db ? da : a.cost > b.cost;
    });
    for (const Group& g : list) {
      const kr_model_desc& d = descs[g.model];
      const int full = d.n_w / cfg->tile_w;
      const int r0 = g.last ? full : 0, r1 = g.last ? full + 1 : full;
      for (int j = 0; j < d.n_p; ++j)
        for (int r = r0; r < r1; ++r)
          *it++ = ItemRec{g.first_pair + j, r * cfg->tile_w,
                          std::min(cfg->tile_w, d.n_w - r * cfg->tile_w), 0};
    }
  };
  write(fwd, reinterpret_cast<ItemRec*>(img + lay.h.off_fwd));
  write(grad, reinterpret_cast<ItemRec*>(img + lay.h.off_grad));
}

extern "C" size_t kr_batch_plan_meta_bytes(const kr_model_desc* descs, int32_t n_models,
                                           const kr_batch_config* cfg) {
  if (!descs || n_models < 0 || !valid_config(cfg)) return 0;
  PlanLayout lay;
  if (layout(descs, n_models, cfg, &lay) != KR_OK) return 0;
  return meta_bytes(lay);
}

extern "C" kr_status kr_batch_plan_host(const kr_model_desc* descs, int32_t n_models,
                                        const kr_batch_config* cfg, void* image,
                                        size_t image_bytes) {
  if (!descs || n_models < 0 || !image) return KR_ERR_INVALID_ARGUMENT;
  if (!valid_config(cfg)) return KR_ERR_INVALID_ARGUMENT;
  PlanLayout lay;
  kr_status s = layout(descs, n_models, cfg, &lay);
  if (s != KR_OK) return s;
  if (image_bytes < meta_bytes(lay)) return KR_ERR_WORKSPACE;
  plan_image(descs, n_models, cfg, lay, static_cast<unsigned char*>(image));
  return KR_OK;
}

extern "C" kr_status kr_batch_plan(const kr_model_desc* descs, int32_t n_models,
                                   const kr_batch_config* cfg, void* plan, size_t plan_bytes,
                                   void* stream) {
  if (!descs || n_models < 0 || !plan) return KR_ERR_INVALID_ARGUMENT;
  if (!valid_config(cfg)) return KR_ERR_INVALID_ARGUMENT;
  PlanLayout lay;
  kr_status s = layout(descs, n_models, cfg, &lay);
  if (s != KR_OK) return s;
  if (plan_bytes < lay.bytes) return KR_ERR_WORKSPACE;
  std::vector<unsigned char> img(meta_bytes(lay));
  plan_image(descs, n_models, cfg, lay, img.data());
  // Pageable source: synchronise before the vector goes out of scope.
  cudaError_t e = cudaMemcpyAsync(plan, img.data(), img.size(), cudaMemcpyHostToDevice,
                                  (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) {
    set_last_error("kr_batch_plan: upload", e);
    return KR_ERR_CUDA;
  }
  return KR_OK;
}

namespace kr {

// One class of the forward items on a resident grid.  `after`: as the programmatic dependent of
// the launch before it (the tangents, or the deep class).
template <int THREADS, ForwardClass CLASS>
static kr_status launch_batch_forward(unsigned char* pl, int max_layers, const double2* w,
                                      double2* R, bool after, cudaStream_t st) {
  const void* fn = (const void*)batch_forward_kernel<THREADS, CLASS>;
  const size_t smem = fwd_smem(THREADS, max_layers, CLASS);
  static SmemLimit lim;
  if (smem > 46 * 1024 &&  // with the static arrays above the 48 KB default
      raise_smem_limit(fn, smem, lim, "kr_batch_launch: forward smem") != KR_OK)
    return KR_ERR_CUDA;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(occupancy_grid(fn, THREADS, smem));
  lc.blockDim = dim3(THREADS);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = after ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&lc, batch_forward_kernel<THREADS, CLASS>, pl, w, R);
  if (e != cudaSuccess) {
    set_last_error("kr_batch_launch: forward", e);
    return KR_ERR_CUDA;
  }
  return KR_OK;
}

// batch_gradient_kernel's shared-memory limit, one for both classes that launch it.
template <int THREADS>
static SmemLimit& gradient_limit() {
  static SmemLimit lim;
  return lim;
}

// One class of the gradient items on a resident grid.  `after`: as the programmatic dependent of
// the class launched before it.
template <int THREADS, bool DEEP>
static kr_status launch_batch_gradient(unsigned char* pl, int max_layers, const double2* w,
                                       const double2* obs, double2* R, double* chi_grad, bool after,
                                       cudaStream_t st) {
  const int L = DEEP ? max_layers : std::min(max_layers, kPqsLayers);
  const size_t sums = batch_sums_enabled() ? sums_smem(THREADS, L) : 0;
  static SmemLimit slim;
  if (!sums) {
    int stage = 0;
    const size_t smem = grad_smem(THREADS, L, &stage);
    const void* fn = (const void*)batch_gradient_kernel<THREADS>;
    if (smem > 46 * 1024 &&
        raise_smem_limit(fn, smem, gradient_limit<THREADS>(), "kr_batch_launch: gradient smem") != KR_OK)
      return KR_ERR_CUDA;
    batch_gradient_kernel<THREADS><<<occupancy_grid(fn, THREADS, smem), THREADS, smem, st>>>(
        pl, w, obs, R, chi_grad, stage, DEEP ? 1 : 0);
    return check_launch("kr_batch_launch: gradient");
  }
  const void* fn = (const void*)batch_grad_sums_kernel<THREADS, DEEP>;
  if (sums > 46 * 1024 &&
      raise_smem_limit(fn, sums, slim, "kr_batch_launch: gradient smem") != KR_OK)
    return KR_ERR_CUDA;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(occupancy_grid(fn, THREADS, sums));
  lc.blockDim = dim3(THREADS);
  lc.dynamicSmemBytes = sums;
  lc.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = after ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&lc, batch_grad_sums_kernel<THREADS, DEEP>, pl, w, obs, R,
                                           chi_grad);
  if (e != cudaSuccess) {
    set_last_error("kr_batch_launch: gradient", e);
    return KR_ERR_CUDA;
  }
  return KR_OK;
}

// One batch launch for a block size of THREADS (32: one warp per work item, i.e. per
// (model, slowness) pair and frequency range; 64 / 128: two / four warps per item).  Grid sizes
// come from occupancy queries (host-side, capture-safe).
template <int THREADS>
static kr_status launch_batch(unsigned char* pl, const kr_batch_config* cfg, int max_layers,
                              const double* layers, const double* p, const double* omega,
                              const double* R_obs, double* R, double* chi_grad,
                              cudaStream_t st) {
  batch_reset_kernel<<<148, 128, 0, st>>>(pl, chi_grad);
  kr_status s = check_launch("kr_batch_launch: reset");
  if (s != KR_OK) return s;
  int gs = 4;
  while (gs < max_layers && gs < kPrepBlock) gs *= 2;
  batch_prep_kernel<<<148 * 16, kPrepBlock, 0, st>>>(pl, layers, p, gs);
  s = check_launch("kr_batch_launch: prep");
  if (s != KR_OK) return s;
  // a batch without observed data has no gradient models: no tangents, no gradient kernel
  const bool grads = R_obs != nullptr, deep = max_layers > kPqsLayers;
  if (grads) {
    // tangents on a resident-sized grid: every block starts at once and releases the forward
    // kernel, its programmatic dependent
    batch_tan_kernel<<<148 * 4, 64, 0, st>>>(pl, p);
    s = check_launch("kr_batch_launch: tangents");
    if (s != KR_OK) return s;
  }
  const double2* w = reinterpret_cast<const double2*>(omega);
  const double2* obs = reinterpret_cast<const double2*>(R_obs);
  double2* R2 = reinterpret_cast<double2*>(R);
  if (deep) {
    const bool lanes = max_layers > kPairLayers || cfg->tile_w <= 64;
    s = lanes ? launch_batch_forward<THREADS, kDeepLanes>(pl, max_layers, w, R2, grads, st)
              : launch_batch_forward<THREADS, kDeepTable>(pl, max_layers, w, R2, grads, st);
    if (s != KR_OK) return s;
  }
  s = launch_batch_forward<THREADS, kShallow>(pl, max_layers, w, R2, grads || deep, st);
  if (s != KR_OK || !grads) return s;
  if (deep) {
    s = launch_batch_gradient<THREADS, true>(pl, max_layers, w, obs, R2, chi_grad, false, st);
    if (s != KR_OK) return s;
  }
  return launch_batch_gradient<THREADS, false>(pl, max_layers, w, obs, R2, chi_grad, deep, st);
}

}  // namespace kr

extern "C" kr_status kr_batch_launch(void* plan, const kr_batch_config* cfg, int32_t max_layers,
                                     const double* layers, const double* p, const double* omega,
                                     const double* R_obs, double* R, double* chi_grad,
                                     void* stream) {
  if (!plan || !valid_config(cfg) || !layers || !p || !omega) return KR_ERR_INVALID_ARGUMENT;
  if (!aligned16(omega) || (R && !aligned16(R)) || (R_obs && !aligned16(R_obs)))
    return KR_ERR_INVALID_ARGUMENT;
  if (max_layers < 2 || max_layers > kMaxLayers) return KR_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* pl = static_cast<unsigned char*>(plan);
  switch (cfg->threads) {
    case 32:
      return launch_batch<32>(pl, cfg, max_layers, layers, p, omega, R_obs, R, chi_grad, st);
    case 64:
      return launch_batch<64>(pl, cfg, max_layers, layers, p, omega, R_obs, R, chi_grad, st);
    default:
      return launch_batch<128>(pl, cfg, max_layers, layers, p, omega, R_obs, R, chi_grad, st);
  }
}
