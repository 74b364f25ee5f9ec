// sg_refine.cu -- FP64 recomputation of the rows whose split-FP32 sums may
// miss the 1e-6 accuracy target.
//
// The split-FP32 kernel accumulates, per row, G^2 = sum over its j-tiles of
// |FP32 tile sum|^2.  The FP32 rounding of the tile sums (the dominant error
// term: the sub-block sums add into a 256-source tile sum in FP32) and of the
// terms behaves like a random walk of size ~1e-7 G, so a row whose
// acceleration cancels (|a| a few % of its G) can reach a relative error of
// several 1e-6 even though its absolute error is ordinary.  The kernel also
// marks (G = infinity) the rows lying more than 8 H from their i-tile centre,
// whose FP32 tile-relative coordinate is rounded by enough to shift the row
// measurably, and leaves out the near pairs of rows that alone have most of
// several tiles within max(H).  k_merge lists the rows with G > T |a|, and
// those without their near pairs, per set; this file plans, on the device, an FP64 pass
// over exactly those rows (k_fp64 over a device-written work list, so the
// call needs no host round trip and stays graph-capturable) and scatters its
// results over the FP32 ones.
//
// Sets with few listed rows (at most REFINE_LIGHT_ROWS) take another route:
// a tile of 128 rows would hold a handful of them, and each row would walk its
// sources one after another, the near pairs (IEEE division and square root)
// setting the time.  There one warp takes one (row, source chunk) item, its
// lanes striding over the chunk's sources (k_refine_light).
//
// Determinism: the list order within a set depends on the merge's atomics,
// but a row's FP64 sum depends only on its own pairs and on the chunk bounds,
// which depend on the per-set counts alone; chunk sums merge in chunk order.
#include "sg_launch.h"

namespace sg {

constexpr int PLAN_NT = 1024;
constexpr int REFINE_LIGHT_ROWS = 32;     // a set with at most this many listed rows: row-chunk items
// Sources per row-chunk item, at least: a row's near pairs, in a few runs of
// sources, then spread over several warps (2,000 particles from host arrays: 152
// us with 512, 140 with 128).
constexpr int REFINE_LIGHT_MIN_J = 128;
constexpr int REFINE_LIGHT_MAX_CH = 256;  // source chunks per light row, at most
constexpr int MERGE_ROWS = 32;            // rows of a merge unit, one per lane
constexpr int MERGE_WARPS = 16;           // warps that share a merge unit's chunks

// Exclusive block scan of one long long per thread (PLAN_NT threads): shuffles
// inside the warps, then over the warp sums; returns the thread's prefix and
// writes the total to *total.
__device__ long long block_exclusive_scan(long long v, long long *total)
{
    __shared__ long long s[PLAN_NT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long add = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += add;
    }
    if (lane == 31) s[w] = incl;
    __syncthreads();
    long long t = s[lane];  // every warp scans the 32 warp sums
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long add = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += add;
    }
    *total = __shfl_sync(0xffffffffu, t, 31);
    const long long before = w > 0 ? __shfl_sync(0xffffffffu, t, w - 1) : 0;
    __syncthreads();  // s is free for the next scan
    return before + incl - v;
}
static_assert(PLAN_NT == 1024, "the scan of the warp sums takes one warp");

// Sources per refine chunk: at least min_j (the host's choice: 256 sources
// with 128-source tiles, 64 with 64-source tiles for small sets), so a few
// listed rows still spread over many blocks (a listed row can have most of
// its set within its softening length, e.g. a point-mass core, and pay the
// near-pair path, one pair after another, for most sources).
__device__ __forceinline__ int refine_chunks(const SetDesc &S, int tj, int min_j, int nch_global)
{
    const int jtiles = (S.n + tj - 1) / tj;
    const int by_len = max(1, (int)(((long long)jtiles * tj) / min_j));
    return max(1, min(nch_global, min(by_len, max(1, jtiles))));
}

__global__ void __launch_bounds__(PLAN_NT) k_refine_plan(const SetDesc *sets, int nsets,
                                                          const int *rcount, int itile, int tj,
                                                          int min_j, int target, int max_items,
                                                          SetDesc *rsets, WorkItem *items,
                                                          int *nitems, int *nlight,
                                                          int *nunits, int *err)
{
    pdl_enter();
    const int t = threadIdx.x;
    const int per = (nsets + blockDim.x - 1) / blockDim.x;
    const int s0 = min(nsets, t * per), s1 = min(nsets, s0 + per);
    int light_most = REFINE_LIGHT_ROWS;
    auto light = [&](int r) { return r > 0 && r <= light_most; };
    // pass 1: refine tiles, light rows and merge units of this thread's sets
    long long tiles = 0, lrows = 0, ltiles = 0, units = 0;
    for (int s = s0; s < s1; s++) {
        const int r = min(rcount[s], sets[s].ni), nt = (r + itile - 1) / itile;
        if (light(r)) {
            lrows += r;
            ltiles += nt;
        } else {
            tiles += nt;
        }
        units += (r + MERGE_ROWS - 1) / MERGE_ROWS;
    }
    long long total_tiles = 0, total_lrows = 0, total_units = 0;
    block_exclusive_scan(tiles, &total_tiles);
    block_exclusive_scan(lrows, &total_lrows);
    if (total_lrows > REFINE_LIGHT_CAP) {
        // more light rows (of thousands of sets) than row-chunk items: all sets
        // take tiles, which fill the GPU then and for which max_items suffices
        long long more = 0;
        block_exclusive_scan(ltiles, &more);
        total_tiles += more;
        total_lrows = 0;
        light_most = 0;
    }
    long long ubase = block_exclusive_scan(units, &total_units);
    const int nch_global = total_tiles > 0 ? (int)max(1ll, (long long)target / total_tiles) : 1;
    const int nchl_global =
        (int)min((long long)REFINE_LIGHT_MAX_CH, max(1ll, REFINE_LIGHT_CAP / max(1ll, total_lrows)));
    auto light_chunks = [&](const SetDesc &S) {
        return max(1, min(nchl_global, S.n / REFINE_LIGHT_MIN_J));
    };
    // pass 2: items of this thread's sets
    long long cnt = 0, lcnt = 0;
    for (int s = s0; s < s1; s++) {
        const int r = min(rcount[s], sets[s].ni);
        if (light(r)) lcnt += (long long)r * light_chunks(sets[s]);
        else cnt += (long long)((r + itile - 1) / itile) * refine_chunks(sets[s], tj, min_j, nch_global);
    }
    long long total_items = 0, total_light = 0;
    long long base = block_exclusive_scan(cnt, &total_items);
    long long lbase = block_exclusive_scan(lcnt, &total_light);
    if (total_items > max_items || total_light > REFINE_LIGHT_CAP) {
        if (t == 0) {
            atomicOr(err, DEVERR_INPUT);
            *nitems = 0;
            *nlight = 0;
            *nunits = 0;
        }
        return;
    }
    // pass 3: the refine descriptors of this thread's sets (slot_off = the
    // set's first tile item, light_off its first row-chunk item, tile_off its
    // first merge unit)
    for (int s = s0; s < s1; s++) {
        SetDesc S = sets[s];
        const int r = min(rcount[s], S.ni);
        const bool lt = light(r);
        const int nt = lt ? 0 : (r + itile - 1) / itile;
        const int nch = refine_chunks(S, tj, min_j, nch_global);
        S.ni = r;
        S.ntiles = nt;
        S.tile_off = (int)ubase;
        ubase += (r + MERGE_ROWS - 1) / MERGE_ROWS;
        S.nchunks = nch;
        S.slot_off = (int)base;
        S.light_off = (int)lbase;
        S.light_nch = lt ? light_chunks(S) : 0;
        rsets[s] = S;
        base += (long long)nt * nch;
        lbase += lt ? (long long)r * S.light_nch : 0;
    }
    __syncthreads();  // rsets visible to the whole block
    // pass 4: the items, spread over all threads (one set can own them all):
    // item k belongs to the last set whose slot_off <= k (a set without
    // items has the slot_off of the next set that has some, so the last
    // such set is never empty)
    for (long long k = t; k < total_items; k += blockDim.x) {
        int lo = 0, hi = nsets - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (rsets[mid].slot_off <= k) lo = mid; else hi = mid - 1;
        }
        const SetDesc S = rsets[lo];
        const int local = (int)(k - S.slot_off);
        const int it = local / S.nchunks, c = local - it * S.nchunks;
        const int jtiles = (S.n + tj - 1) / tj;
        WorkItem w;
        w.set = lo;
        w.tile = it;
        w.chunk = c;
        w.slot = (int)k;  // = S.slot_off + it * S.nchunks + c
        w.jb = (int)((long long)jtiles * c / S.nchunks) * tj;
        w.je = (int)((long long)jtiles * (c + 1) / S.nchunks) * tj;
        w.pad_[0] = w.pad_[1] = 0;
        items[k] = w;
    }
    if (t == 0) {
        *nitems = (int)total_items;
        *nlight = (int)total_light;
        *nunits = (int)total_units;
    }
}

// One warp per (listed row, source chunk) item of a light set: lanes stride
// over the chunk's sources, 32 steps to a mask.  Newtonian pairs go straight
// into the lane's sums; the pairs that may be near are flagged and then
// evaluated with the CPU path's formulas one per lane (a step with one near
// pair would cost the warp as much as 32 of them).  A fixed butterfly sums the
// lanes; lpart[item][4] receives the chunk's sums.
__global__ void __launch_bounds__(256) k_refine_light(const SetDesc *rsets, int nsets,
                                                     const int *nitems, const int *rlist,
                                                     SortedF64 D, int nkernel, double *lpart)
{
    constexpr unsigned FULL = 0xffffffffu;
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int n_it = *nitems;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < n_it; k += nw) {
        // item k: the last set whose light_off is at most k (sets without items
        // share the offset of the next one that has some), its row and chunk
        int lo = 0, hi = nsets - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (rsets[mid].light_off <= k) lo = mid; else hi = mid - 1;
        }
        const SetDesc S = rsets[lo];
        const int row = (k - S.light_off) / S.light_nch;
        const int c = k - S.light_off - row * S.light_nch;
        const int jb = S.poff + (int)((long long)S.n * c / S.light_nch);
        const int je = S.poff + (int)((long long)S.n * (c + 1) / S.light_nch);
        const int i = rlist[S.ioff + row];
        const double xi = D.x[i], yi = D.y[i], zi = D.z[i], hi2 = D.h2[i];
        const int hih = __double2hiint(hi2);
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        for (int j0 = jb; j0 < je; j0 += 1024) {
            const int cnt = min(32, (je - j0 + 31) / 32);
            uint32_t m = 0u;
#pragma unroll 4
            for (int u = 0; u < cnt; u++) {
                const int j = j0 + 32 * u + lane;
                if (j < je) {
                    const double dx = D.x[j] - xi, dy = D.y[j] - yi, dz = D.z[j] - zi;
                    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
                    if (maybe_near(r2, max(hih, __double2hiint(D.h2[j])))) {
                        m |= 1u << u;
                    } else {
                        const double y = rsqrt_f64(r2);
                        const double mr = D.m[j] * y;
                        const double mr3 = mr * (y * y);
                        acc[0] = fma(mr3, dx, acc[0]);
                        acc[1] = fma(mr3, dy, acc[1]);
                        acc[2] = fma(mr3, dz, acc[2]);
                        acc[3] -= mr;
                    }
                }
            }
            const int c = __popc(m);
            const int incl = warp_inclusive(c, lane);
            const int total = __shfl_sync(FULL, incl, 31);
            for (int base = 0; base < total; base += 32) {
                const int g = base + lane;
                const int ow = warp_owner(incl, g);
                const uint32_t mo = __shfl_sync(FULL, m, ow);
                const int eo = __shfl_sync(FULL, incl - c, ow);
                if (g < total) {
                    const int j = j0 + 32 * nth_bit(mo, g - eo) + ow;
                    const PairOut o = pair_f64_core(D, nkernel, i, j, D.x[j] - xi, D.y[j] - yi,
                                                    D.z[j] - zi, D.m[j], hi2, D.h2[j]);
                    acc[0] += o.ax;
                    acc[1] += o.ay;
                    acc[2] += o.az;
                    acc[3] += o.pot;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(FULL, acc[q], o);
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 4; q++) lpart[(size_t)k * 4 + q] = acc[q];
        }
    }
}

cudaError_t launch_refine_light(const SetDesc *rsets, int nsets, const int *nitems,
                                const int *rlist, const SortedF64 &D, int nkernel, double *lpart,
                                int sm_count, cudaStream_t st)
{
    return launch(k_refine_light, sm_count * 8, 256, 0, st, rsets, nsets, nitems, rlist, D, nkernel,
                  lpart);
}

cudaError_t launch_refine_plan(const SetDesc *sets, int nsets, const int *rcount, int itile,
                               int tj, int min_j, int target, int max_items, SetDesc *rsets,
                               WorkItem *items, int *nitems, int *nlight, int *nunits, int *err,
                               cudaStream_t st)
{
    return launch(k_refine_plan, 1, PLAN_NT, 0, st, sets, nsets, rcount, itile, tj, min_j, target,
                  max_items, rsets, items, nitems, nlight, nunits, err);
}

// Scatter of the refined rows, by units of MERGE_ROWS listed rows: lane = row,
// so the loads of a tile item's sums are coalesced, and the block's warps share
// the item's chunks; the warps' sums add in order (deterministic).  Bound by
// the latency of those loads: a few tiles of rows have up to ~1,000 chunks
// each.  One warp per row, 4 warps per main i-tile, took 731 us for one rank's
// 15,309 rows of a 61,237-particle collision (its ~200 listed rows all in the
// first i-tile's block, 8 of each 32 bytes loaded used).
__global__ void __launch_bounds__(MERGE_WARPS * 32)
k_refine_merge(const SetDesc *rsets, int nsets, const int *nunits, int itile_ref,
               const int *rlist, SortedF64 D, const double *rpart, const double *lpart,
               OutputsDev out)
{
    __shared__ double s_sum[MERGE_WARPS][4][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_enter();
    const int nu = *nunits;
    for (int u = blockIdx.x; u < nu; u += gridDim.x) {
        // the last set whose first unit is <= u (sets without units share the
        // offset of the next set that has some)
        int lo = 0, hi = nsets - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (rsets[mid].tile_off <= u) lo = mid; else hi = mid - 1;
        }
        const SetDesc RS = rsets[lo];
        const int li = (u - RS.tile_off) * MERGE_ROWS + lane;
        const bool act = li < RS.ni;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        if (act && RS.light_nch > 0) {  // row-chunk items
            const double *p = lpart + (size_t)(RS.light_off + li * RS.light_nch) * 4;
#pragma unroll 4
            for (int c = warp; c < RS.light_nch; c += MERGE_WARPS) {
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q] += p[(size_t)c * 4 + q];
            }
        } else if (act) {
            const int rt = li / itile_ref, ri = li - rt * itile_ref;
            const double *p = rpart + (size_t)(RS.slot_off + rt * RS.nchunks) * 4 * itile_ref + ri;
#pragma unroll 4
            for (int c = warp; c < RS.nchunks; c += MERGE_WARPS) {
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q] += p[((size_t)c * 4 + q) * itile_ref];
            }
        }
        __syncthreads();  // the previous unit's sums have been read
#pragma unroll
        for (int q = 0; q < 4; q++) s_sum[warp][q][lane] = acc[q];
        __syncthreads();
        if (warp < 4 && act) {  // warp q: quantity q
            double v = s_sum[0][warp][lane];
#pragma unroll
            for (int w = 1; w < MERGE_WARPS; w++) v += s_sum[w][warp][lane];
            double *dst = warp == 0 ? out.ax : warp == 1 ? out.ay : warp == 2 ? out.az : out.pot;
            dst[D.orig[rlist[RS.ioff + li]]] = v;
        }
    }
}

cudaError_t launch_refine_merge(const SetDesc *rsets, int nsets, const int *nunits, int itile_ref,
                                const int *rlist, const SortedF64 D, const double *rpart,
                                const double *lpart, OutputsDev out, int sm_count, cudaStream_t st)
{
    return launch(k_refine_merge, 2 * sm_count, MERGE_WARPS * 32, 0, st, rsets, nsets, nunits,
                  itile_ref, rlist, D, rpart, lpart, out);
}

}  // namespace sg
