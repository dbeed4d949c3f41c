// force.cu -- the i-block x j-particle direct-summation kernel.
//
// Pair terms are those of the reference's accumulate_acc_and_jerk
// (src/node/dyn/hdyn/evolve/hdyn_ev.C:2019-2036): with dr = x_j - x_i,
// dv = v_j - v_i, r2 = dr.dr + eps2,
//     pot -= m/r,  acc += m dr / r^3,  jerk += m/r^3 (dv - 3 (dr.dv)/r2 dr),
// self excluded by index; the nearest neighbour is the first address with
// the smallest dr.dr (no softening; hdyn_inline.C:34-77).
//
// GRAPE-4 variant (FP64 only, kVarG4): the pipeline of the reference's
// GRAPE-4 simulator (src/harpsims/harp3fastsim.c:240-300): per-i softening,
// r2 = dr.dr + eps2_i; a pair contributes only when r2 > 0 (no exclusion by
// index: kira stores the block's own particles at the block time, so self
// has dr = 0 exactly); neighbour test r2 < h2_i on the softened r2.
//
// Work decomposition (one launch):
//   gridDim.x  i-tiles;  gridDim.y  j-splits (contiguous address ranges,
//              whole tiles; the last CTA of an i-tile adds their partial
//              sums in a fixed order, so the result is deterministic);
//   CTA        NW warps = G i-groups x H j-subranges;
//   warp       IL i-lanes x JL = 32/IL j-lanes; each thread owns R i's
//              (register blocking: each j read from shared memory feeds R
//              pair evaluations).
// j-tiles of T records move global -> shared by one bulk copy (TMA,
// cp.async.bulk + mbarrier) per tile, double-buffered: the copy of tile t+1
// is in flight while tile t is consumed.  Partial sums over the JL j-lanes
// are combined with warp shuffles (xor butterfly, identical on every lane),
// then over the H warps through shared memory.
//
// Mixed mode pair arithmetic is FP32 (exact position differences from the
// fixed-point positions, Newton-refined rsqrt.approx); each thread sums up
// to kFlush pair terms in FP32 and then folds them into FP64 totals.  The
// paired layout evaluates two j per FP32x2 instruction (add/mul/fma.f32x2),
// halving the issue slots per interaction.  FP64 mode does the pair
// arithmetic and the sums in FP64.
#include <algorithm>
#include <cfloat>
#include "common.cuh"
#include "force_device.cuh"
#include "kernels.h"

namespace g6 {


int tile_size(int kmode) { return kmode == kKernF64 ? Traits<kKernF64>::T : 256; }

static int units_per_tile(int kmode) { return kmode == kKernMixedP ? Traits<kKernMixedP>::U : tile_size(kmode); }

size_t jrec_bytes(int kmode) {
    switch (kmode) {
        case kKernF64: return sizeof(JRecF64);
        case kKernMixedP: return sizeof(JPairMixed) / 2;
        default: return sizeof(JRecMixed);
    }
}

// ----------------------------------------------------------------------------

// One call: gridDim.x i-tiles x gridDim.y j-splits, one task per CTA.
template <int K, int IL, int R, bool NB, bool IDENT, int V>
__global__ void __launch_bounds__(256, MinBlocks<K, R>::value) force_kernel(const ForceParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    init_bars(smem);
    if (p.status_clear && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *p.status_clear = 0u;
    int gt = 0;
    process_task<K, IL, R, NB, IDENT, V>(p, blockIdx.x, blockIdx.y, smem, gt);
}

// A small FP64 call in one launch: its staged updates to the raw j-state,
// the prediction of each CTA's j-range, the forces (process_task's JFromCall
// form).  As two launches (updates and prediction, then forces) a block of
// 61 against 40009 j took 14.2 + 30.0 us on the device, one of 24 against
// 1024 10.5 + 9.5; as one 23.3 and 10.5.
template <int IL, bool NB, bool IDENT, int V>
__global__ void __launch_bounds__(256, 1)
    small_force_kernel(const __grid_constant__ SmallCall param, ForceParams p, double *jraw, int *jindex,
                       unsigned *status2) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_addr[kSmallMax];
    const SmallCall &sc = param_as_memory(param);
    if (threadIdx.x < sc.n_upd) s_addr[threadIdx.x] = sc.addr[threadIdx.x];
    const int cta = blockIdx.x + gridDim.x * blockIdx.y;
    if (cta == 0 && threadIdx.x == 0) status2[sc.parity ^ 1] = 0u;
    store_updates(sc, cta, gridDim.x * gridDim.y, jraw, jindex);
    p.irec = sc.irec;
    p.ieps2 = sc.g4 ? sc.ieps2 : nullptr;
    __syncthreads();
    int gt = 0;
    process_task<kKernF64, IL, 1, NB, IDENT, V, JFromCall>(p, blockIdx.x, blockIdx.y, smem, gt,
                                                           JFromCall{&sc, jraw, jindex, s_addr});
}

// Many calls in one launch: items[k] is one call (its own j-memory,
// i-records, softening, fixed-point scale and outputs); its tasks are
// n_itiles(k) x nsplit(k), numbered from task0[k].  Persistent form: CTAs
// take tasks from a global counter until the list is exhausted.  With
// one_task_per_cta, CTA b runs task b (so CTAs of other launches can be
// scheduled as these retire).
template <int K, int IL, int R, bool NB, bool IDENT, int V>
__global__ void __launch_bounds__(256, MinBlocks<K, R>::value) batch_force_kernel(const BatchArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_task;
    init_bars(smem);
    const int itile = (blockDim.x >> 5) / a.H * IL * R;
    const int total = a.task0[a.n_items];
    int gt = 0;
    for (int it = 0;; ++it) {
        __syncthreads();
        if (threadIdx.x == 0) s_task = a.one_task_per_cta ? (it == 0 ? (int)blockIdx.x : total) : atomicAdd(a.counter, 1);
        __syncthreads();
        const int task = s_task;
        if (task >= total) break;
        int lo = 0, hi = a.n_items - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.task0[mid] <= task) lo = mid; else hi = mid - 1;
        }
        const ForceParams p = a.items[a.order ? a.order[lo] : lo];
        const int local = task - a.task0[lo];
        const int il = batch_il(p.ni);  // the item's lane shape (its H is in p.H)
        bool ok;
        if (il == 32) {
            const int n_itiles = (p.ni + itile - 1) / itile;
            ok = process_task<K, IL, R, NB, IDENT, V>(p, local % n_itiles, local / n_itiles, smem, gt);
        } else if (il == 8) {
            const int it8 = (blockDim.x >> 5) / p.H * 8;
            const int n_itiles = (p.ni + it8 - 1) / it8;
            ok = process_task<K, 8, 1, NB, IDENT, V>(p, local % n_itiles, local / n_itiles, smem, gt);
        } else {
            const int it1 = (blockDim.x >> 5) / p.H;
            const int n_itiles = (p.ni + it1 - 1) / it1;
            ok = process_task<K, 1, 1, NB, IDENT, V>(p, local % n_itiles, local / n_itiles, smem, gt);
        }
        // After a timed-out copy wait this CTA's barrier phases no longer
        // match its tile count: it takes no further task (the status word
        // already reports the failure; the other CTAs finish the list).
        if (!ok) break;
    }
}

// Split reduction for every i of every item with nsplit > 1; ipre[k] is the
// prefix sum of the items' ni (read on the device, so a launch captured in a
// graph serves batches of any size: grid-stride over ipre[n_items]).
__global__ void batch_reduce_kernel(const BatchArgs a) {
    const int total = a.ipre[a.n_items];
    for (int gi = blockIdx.x * blockDim.x + threadIdx.x; gi < total; gi += gridDim.x * blockDim.x) {
        int lo = 0, hi = a.n_items - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.ipre[mid] <= gi) lo = mid; else hi = mid - 1;
        }
        const ForceParams &p = a.items[lo];
        if (p.nsplit <= 1) continue;
        const int i = gi - a.ipre[lo];
        Partial q = p.part[i];
        for (int s = 1; s < p.nsplit; ++s) add_partial(q, p.part[(size_t)s * p.ni + i]);
        write_final(p, i, q);
    }
}

__global__ void reduce_partials_kernel(const ForceParams p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.ni) return;
    Partial a = p.part[i];
    for (int s = 1; s < p.nsplit; ++s) add_partial(a, p.part[(size_t)s * p.ni + i]);
    write_final(p, i, a);
}

// ----------------------------------------------------------------------------
// Host side: kernel selection and launch geometry.

using KernelFn = void (*)(const ForceParams);

template <int K, int IL, int R>
static KernelFn pick3(bool nb, bool ident) {
    // the single-call paired mixed kernels also accumulate the refinement's
    // error indicators
    constexpr int V = kVarUnroll4 | (K == kKernMixedP ? kVarStats : 0);
    if (nb) return ident ? force_kernel<K, IL, R, true, true, V> : force_kernel<K, IL, R, true, false, V>;
    return ident ? force_kernel<K, IL, R, false, true, V> : force_kernel<K, IL, R, false, false, V>;
}

template <int K>
static KernelFn pick2(int il, int r, bool nb, bool ident) {
    if (il == 32) {
        if constexpr (K == kKernMixedDS) {
            if (r == 4) return pick3<K, 32, 4>(nb, ident);
        }
        if constexpr (K != kKernMixedP) {
            if (r == 2) return pick3<K, 32, 2>(nb, ident);
        }
        return pick3<K, 32, 1>(nb, ident);
    }
    if (il == 8) return pick3<K, 8, 1>(nb, ident);
    return pick3<K, 1, 1>(nb, ident);
}

// GRAPE-4 pipeline: FP64 layout, no index identity.
static KernelFn pick_g4(int il, int r, bool nb) {
    constexpr int K = kKernF64, V = kVarG4;
    if (il == 32 && r == 2) return nb ? force_kernel<K, 32, 2, true, false, V> : force_kernel<K, 32, 2, false, false, V>;
    if (il == 32) return nb ? force_kernel<K, 32, 1, true, false, V> : force_kernel<K, 32, 1, false, false, V>;
    if (il == 8) return nb ? force_kernel<K, 8, 1, true, false, V> : force_kernel<K, 8, 1, false, false, V>;
    return nb ? force_kernel<K, 1, 1, true, false, V> : force_kernel<K, 1, 1, false, false, V>;
}

// Potential only (energy sweeps): one i per thread, no neighbour lists.
template <int K>
static KernelFn pick_pot(int il, bool ident) {
    constexpr int V = kVarUnroll4 | kVarPot;
    if (il == 32) return ident ? force_kernel<K, 32, 1, false, true, V> : force_kernel<K, 32, 1, false, false, V>;
    if (il == 8) return ident ? force_kernel<K, 8, 1, false, true, V> : force_kernel<K, 8, 1, false, false, V>;
    return ident ? force_kernel<K, 1, 1, false, true, V> : force_kernel<K, 1, 1, false, false, V>;
}

static KernelFn pick(int kmode, int il, int r, bool nb, bool ident) {
    if (kmode == kKernMixedP) return pick2<kKernMixedP>(il, r, nb, ident);
    if (kmode == kKernMixedDS) return pick2<kKernMixedDS>(il, r, nb, ident);
    return pick2<kKernF64>(il, r, nb, ident);
}

static size_t smem_bytes(int kmode, const ForceConfig &c) {
    size_t tiles = 2 * (size_t)tile_size(kmode) * jrec_bytes(kmode);  // bytes per j x j per tile
    size_t itile = (size_t)(c.warps / c.H) * c.il * c.r;
    size_t red = c.H > 1 ? (size_t)c.H * itile * sizeof(Partial) : 0;
    return 128 + (tiles > red ? tiles : red);
}

size_t partial_bytes(const ForceConfig &cfg, int ni) {
    return cfg.nsplit > 1 ? (size_t)cfg.nsplit * ni * sizeof(Partial) : 0;
}

size_t partial_bytes_fixed(int jper, int nj_pad, int ni) {
    const int nsplit = std::max(1, (nj_pad + jper - 1) / jper);
    return (size_t)nsplit * ni * sizeof(Partial);
}

// The shape from ni, the splits from a fill rule: blocks of up to 64 i (the
// i-lane shapes, and the one-launch kernel with its one CTA per SM), the
// scalar mixed layout, and j-split calls, whose sums must not depend on the
// size of a rank's slice.
ForceConfig fill_config(int kmode, int ni, int nj_pad, int num_sms) {
    ForceConfig c;
    c.warps = kMaxWarps;
    c.il = ni >= 32 ? 32 : (ni > 1 ? 8 : 1);
    if (c.il == 8 && ni > 8) c.il = 32;
    // Register blocking: the scalar mixed layout gains from 2 i per thread,
    // and so does FP64 (two independent FP64 chains per thread hide part of
    // the dependency waits: 9.40 vs 9.56 ms for 16384 x 262144); the
    // paired layout already reuses each loaded j-pair twice and runs out of
    // registers at 2 (measured: 91 ms vs 95 ms for the N = 262144 sweep).
    c.r = ((kmode == kKernMixedDS || kmode == kKernF64) && c.il == 32 && ni >= 8192) ? 2 : 1;
    // i-groups per CTA: at most an eighth of the i-block per CTA, so that a
    // mid-size block spreads over several i-tiles instead of one i-tile
    // split many ways, whose split fold then dominates.  Measured at nj =
    // 262144 (mixed, with one thread per i over all splits; fold_splits has
    // shortened the fold since): ni = 256 0.12 vs 0.31 ms, ni = 1024 0.39 vs
    // 0.43 ms; ni >= 2048 unchanged (8 groups).
    int groups_needed = (ni + c.il * c.r - 1) / (c.il * c.r);
    int G = 1;
    while (G * 2 <= c.warps && G * 2 * 8 <= groups_needed) G *= 2;
    c.H = c.warps / G;
    const int T = tile_size(kmode);
    const int JL = 32 / c.il;
    const int U = units_per_tile(kmode);
    while (c.H > 1 && U / (c.H * JL) < 1) c.H /= 2;  // keep >= 1 record per thread per tile
    G = c.warps / c.H;
    const int itile = G * c.il * c.r;
    const int n_itiles = (ni + itile - 1) / itile;
    const int ntiles = nj_pad / T;
    // Fill the GPU with whole waves: 2 resident CTAs per SM, or one per SM
    // for blocks of up to 128 i (fewer splits to fold: ni = 64 0.051 vs
    // 0.062 ms, ni = 16 0.042 vs 0.058 ms).
    const int slots = (ni <= 128 ? 1 : 2) * num_sms;
    int best_split = 1;
    double best_eff = -1;
    for (int sp = 1; sp <= ntiles && sp <= 4096; ++sp) {
        const int per_split_tiles = (ntiles + sp - 1) / sp;
        const int real_split = (ntiles + per_split_tiles - 1) / per_split_tiles;
        if (real_split != sp) continue;
        const long long ctas = (long long)n_itiles * sp;
        const long long waves = (ctas + slots - 1) / slots;
        double eff = (double)ctas / (double)(waves * slots);
        // Penalise tiny per-CTA work (tile pipeline start-up, reduction).
        if (per_split_tiles < 4 && sp > 1) eff *= 0.5;
        if (eff > best_eff + 1e-9) {
            best_eff = eff;
            best_split = sp;
        }
        if (ctas >= 8LL * slots) break;
    }
    c.nsplit = best_split;
    return c;
}

// Predicted time (us) of a call's force kernel for a launch shape: fitted to
// 8000 measured launches (ni 65 to 20096, nj 1024 to 262144, every r and H,
// up to 24 CTAs per SM).  80 % of the FP64 times lie within -10 and +6 % of
// it, of the mixed ones within 3 %; the shape it picks is on average 0.4 %
// (mixed 0.7 %) slower than the best one measured, at worst 5 %.  Filling
// the SMs' slots with whole waves instead -- which takes a full wave however
// little work its CTAs then have -- was up to 1.7 times slower than the best
// (kernel alone: mixed 2048 x 20096 0.129 against 0.075 ms, FP64 2048 x 20096
// 0.131 against 0.111, 1024 x 4096 0.027 against 0.021).
//   step   j-steps (records) of the two warps of one CTA on a scheduler
//   k      CTAs the busiest SM runs, two at a time; an odd last one is alone.
//          A grid of up to one CTA per SM is counted as two on some: launched
//          back to back it is spread evenly, in calls it was not (2000 x
//          262144 in 126 CTAs 1.44 ms a call, in 296 1.40).
struct ShapeCost {
    double base, step, alone, cta, tile, round, level;
};
constexpr ShapeCost kCostF64{6.3, 0.0427, 0.0034, 2.15, 0.082, 0.96, 0.90};
constexpr ShapeCost kCostMixed{12.5, 0.0512, 0.0033, 0.0, 0.224, 1.53, 1.10};

static double shape_cost(const ShapeCost &q, int kmode, const ForceConfig &c, int ni, int ntiles, int num_sms) {
    const int itile = c.warps / c.H * c.il * c.r;
    const int n_itiles = (ni + itile - 1) / itile;
    const int per = (ntiles + c.nsplit - 1) / c.nsplit;
    const int k = std::max(2, (int)(((long long)n_itiles * c.nsplit + num_sms - 1) / num_sms));
    const double step = (double)per * (units_per_tile(kmode) / c.H) * 2 * c.r;
    double t = q.base + q.step * k * step + q.cta * k + q.tile * per * ((k + 1) / 2);
    if (k & 1) t += q.alone * step;
    if (c.nsplit > 1) {  // the fold: fold_splits' segments, rounds of four loads, pairwise levels
        int it2 = 1, segs = 1;
        while (it2 < itile) it2 <<= 1;
        for (; 2 * segs * it2 <= 32 * c.warps && 8 * segs < c.nsplit; segs <<= 1) t += q.level;
        t += q.round * ((c.nsplit + segs - 1) / segs) * 0.25 * ((itile + 32 * c.warps - 1) / (32 * c.warps));
    }
    return t;
}

ForceConfig choose_config(int kmode, int ni, int nj_pad, int num_sms, bool nb) {
    (void)nb;
    const ForceConfig fill = fill_config(kmode, ni, nj_pad, num_sms);
    const int ntiles = nj_pad / tile_size(kmode);
    if (ni <= 64 || ntiles <= 1 || kmode == kKernMixedDS) return fill;
    const ShapeCost &q = kmode == kKernF64 ? kCostF64 : kCostMixed;
    ForceConfig best = fill;
    // the whole waves stay unless 4 % or more is expected: their last wave is
    // full, which a grid of a few long CTAs does not always achieve
    double least = 0.96 * shape_cost(q, kmode, fill, ni, ntiles, num_sms);
    for (int r = 1; r <= (kmode == kKernF64 ? 2 : 1); ++r)
        for (int H = 1; H <= fill.warps; H *= 2) {
            // The mixed mode sums 64 terms in FP32: with H of 1, 2 or 4 the
            // same 32 records of a tile, with 8 halves of them.  A block's
            // results keep to the one its size had.
            if (kmode == kKernMixedP && (H == fill.warps) != (fill.H == fill.warps)) continue;
            ForceConfig c = fill;
            c.r = r;
            c.H = H;
            const int itile = c.warps / H * c.il * r;
            const int n_itiles = (ni + itile - 1) / itile;
            int last = 0;
            for (int k = 1; k <= 12; ++k) {  // splits that give the busiest SM k CTAs
                const int want = std::min(std::max(1, (int)((long long)num_sms * k / n_itiles)), ntiles);
                const int per = (ntiles + want - 1) / want;
                c.nsplit = (ntiles + per - 1) / per;
                if (c.nsplit == last) continue;
                last = c.nsplit;
                const double t = shape_cost(q, kmode, c, ni, ntiles, num_sms);
                if (t < least) {
                    least = t;
                    best = c;
                }
            }
        }
    return best;
}

// ---- batched (multi-item persistent) launches

using BatchFn = void (*)(const BatchArgs);

template <int K>
static BatchFn pick_batch(bool nb, bool ident) {
    constexpr int V = kVarUnroll4;
    if (nb) return ident ? batch_force_kernel<K, 32, 1, true, true, V> : batch_force_kernel<K, 32, 1, true, false, V>;
    return ident ? batch_force_kernel<K, 32, 1, false, true, V> : batch_force_kernel<K, 32, 1, false, false, V>;
}

static BatchFn pick_batch(int kmode, bool nb, bool ident) {
    if (kmode == kKernMixedP) return pick_batch<kKernMixedP>(nb, ident);
    if (kmode == kKernMixedDS) return pick_batch<kKernMixedDS>(nb, ident);
    return pick_batch<kKernF64>(nb, ident);
}

ForceConfig batch_config(int kmode) {
    (void)kmode;
    ForceConfig c;
    c.il = 32;
    c.r = 1;
    c.warps = kMaxWarps;
    c.H = 4;
    c.nsplit = 0;
    return c;
}

int batch_ctas(int kmode, const ForceConfig &cfg, int num_sms) {
    int per_sm = 0;
    BatchFn fn = pick_batch(kmode, false, true);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * cfg.warps, smem_bytes(kmode, cfg));
    if (per_sm < 1) per_sm = 1;
    return per_sm * num_sms;
}

cudaError_t launch_force_batch(cudaStream_t s, int kmode, const ForceConfig &cfg, const BatchArgs &a, int ctas,
                               int total_i, bool nb, bool ident) {
    if (a.n_items <= 0) return cudaSuccess;
    BatchFn fn = pick_batch(kmode, nb, ident);
    fn<<<ctas, 32 * cfg.warps, smem_bytes(kmode, cfg), s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (total_i > 0) {
        batch_reduce_kernel<<<std::min((total_i + 255) / 256, 1184), 256, 0, s>>>(a);
        e = cudaGetLastError();
    }
    return e;
}

// Fills jper, nsplit and H of p as launch_force does, and returns its i-tile.
static int plan_call(int kmode, const ForceConfig &cfg, ForceParams &p) {
    const int T = tile_size(kmode), ntiles = p.nj_pad / T;
    if (ntiles <= 0) {
        p.jper = T;
        p.nsplit = 1;
    } else {
        const int per_split_tiles = (ntiles + cfg.nsplit - 1) / cfg.nsplit;
        p.jper = per_split_tiles * T;
        p.nsplit = (ntiles + per_split_tiles - 1) / per_split_tiles;
    }
    p.H = cfg.H;
    return cfg.warps / cfg.H * cfg.il * cfg.r;
}

using SmallFn = void (*)(const SmallCall, ForceParams, double *, int *, unsigned *);

template <int IL>
static SmallFn pick_small(bool nb, bool ident, bool g4) {
    constexpr int V = kVarUnroll4;
    if (g4) return nb ? small_force_kernel<IL, true, false, kVarG4> : small_force_kernel<IL, false, false, kVarG4>;
    if (nb) return ident ? small_force_kernel<IL, true, true, V> : small_force_kernel<IL, true, false, V>;
    return ident ? small_force_kernel<IL, false, true, V> : small_force_kernel<IL, false, false, V>;
}

static SmallFn pick_small(int il, bool nb, bool ident, bool g4) {
    return il == 32 ? pick_small<32>(nb, ident, g4) : il == 8 ? pick_small<8>(nb, ident, g4)
                                                              : pick_small<1>(nb, ident, g4);
}

static size_t small_smem_bytes(const ForceConfig &cfg, const ForceParams &p, int itile) {
    const size_t j = (size_t)p.jper * sizeof(JRecF64);
    const size_t red = std::max((size_t)cfg.H * itile, (size_t)16 * cfg.warps) * sizeof(Partial);
    return 128 + std::max(j, red);
}

bool small_force_fits(const ForceConfig &cfg, ForceParams p) {
    const int itile = plan_call(kKernF64, cfg, p);
    return cfg.r == 1 && cfg.H > 1 && p.nj_pad > 0 && small_smem_bytes(cfg, p, itile) <= kSmallSmemMax;
}

int small_force_variant(const ForceConfig &cfg, bool ident, bool nb, bool g4) {
    return 6 * (cfg.il == 32 ? 0 : cfg.il == 8 ? 1 : 2) + (g4 ? 4 + nb : 2 * ident + nb);
}

cudaError_t prepare_small_force(int variant) {
    const int il = variant / 6 == 0 ? 32 : variant / 6 == 1 ? 8 : 1, v = variant % 6;
    return cudaFuncSetAttribute(pick_small(il, v & 1, v & 2, v >= 4), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSmallSmemMax);
}

cudaError_t launch_small_force(cudaStream_t s, const ForceConfig &cfg, ForceParams p, const SmallCall &sc,
                               double *jraw, int *jindex, unsigned *status2, bool ident, bool nb) {
    const int itile = plan_call(kKernF64, cfg, p);
    const dim3 grid((p.ni + itile - 1) / itile, p.nsplit);
    pick_small(cfg.il, nb, ident, sc.g4 != 0)<<<grid, 32 * cfg.warps, small_smem_bytes(cfg, p, itile), s>>>(
        sc, p, jraw, jindex, status2);
    return cudaGetLastError();
}

cudaError_t launch_force(cudaStream_t s, int kmode, const ForceConfig &cfg, ForceParams p,
                         bool ident, bool nb, bool g4, bool pot) {
    if (g4 && (kmode != kKernF64 || !p.ieps2)) return cudaErrorInvalidValue;
    if (pot && (g4 || nb || cfg.r != 1 || kmode == kKernMixedDS)) return cudaErrorInvalidValue;
    const int T = tile_size(kmode);
    if (p.ni <= 0) return cudaSuccess;
    const int itile = plan_call(kmode, cfg, p);
    if (cfg.jper > 0) {
        if (cfg.jper % T) return cudaErrorInvalidValue;
        p.jper = cfg.jper;
        p.nsplit = std::max(1, (p.nj_pad + cfg.jper - 1) / cfg.jper);
    }
    dim3 grid((p.ni + itile - 1) / itile, p.nsplit);
    dim3 block(32 * cfg.warps);
    KernelFn fn = pot ? (kmode == kKernF64 ? pick_pot<kKernF64>(cfg.il, ident) : pick_pot<kKernMixedP>(cfg.il, ident))
                      : g4 ? pick_g4(cfg.il, cfg.r, nb) : pick(kmode, cfg.il, cfg.r, nb, ident);
    size_t sm = smem_bytes(kmode, cfg);
    fn<<<grid, block, sm, s>>>(p);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (p.nsplit > 1 && !p.tile_counter && !p.keep_partials) {
        reduce_partials_kernel<<<(p.ni + 255) / 256, 256, 0, s>>>(p);
        e = cudaGetLastError();
    }
    return e;
}

// Self-test of the bounded wait that guards every j-tile copy: one thread
// waits on an mbarrier that nothing arrives at and no copy completes, so
// the wait runs out after limit_ns and the status word gets the same bit a
// force call sets when a copy wait times out.  No copy is in flight when it
// gives up.
__global__ void copy_wait_selftest_kernel(unsigned *status, unsigned long long limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    fence_barrier_init();
    if (!mbar_wait_bounded(&bar, 0, limit_ns)) atomicOr(status, ST_TMA_TIMEOUT);
}

void launch_copy_wait_selftest(cudaStream_t s, unsigned *status, unsigned long long limit_ns) {
    copy_wait_selftest_kernel<<<1, 32, 0, s>>>(status, limit_ns);
}

}  // namespace g6
