// sg_launch.h -- host-side launch interface between the context code and the
// kernels.  Every function enqueues on `st` and returns the launch status.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <atomic>
#include "sg_internal.cuh"

namespace sg {

// Kernels launched by the library; atomic because entry points on different
// contexts (or the allocation-free one) may run on several host threads.
extern std::atomic<unsigned long long> g_launches;

// Launch with programmatic dependence on the stream's previous kernel: the
// blocks may start while that kernel drains, and wait in pdl_wait() until it
// has completed and its writes are visible.  Every kernel launched this way
// calls pdl_enter() (or pdl_wait()) before it touches global memory.
template <class... P, class... A>
inline cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                          A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    ++g_launches;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Kernels with a set per block row loop over the sets that a grid's second
// dimension (at most 65,535) cannot number.
inline unsigned grid_sets(int nsets) { return nsets < 65535 ? nsets : 65535; }

// Input arrays in the caller's (original) order, device pointers.
struct InputsDev {
    const double *x, *y, *z, *m, *r2;
};
// Outputs in the caller's order, device pointers (rows only are written).
struct OutputsDev {
    double *ax, *ay, *az, *pot;
};

// --- preparation (sg_prep.cu)
// Counters that a call's kernels count up from zero.
struct Counters {
    int *head = nullptr, *rhead = nullptr;  // queue heads (rhead nullable)
    int *rcount = nullptr;                  // [nsets] refine rows per set (nullable)
};
// Checks the inputs (DEVERR_INPUT), folds the sets' bounding boxes into bbox
// and zeroes the call's counters.  bbox: 6 words per set, all bits set between
// calls (launch_gather leaves them so): min of dkey(lo), min of ~dkey(hi).
cudaError_t launch_bbox(const SetDesc *sets, int nsets, int max_n, const InputsDev &in,
                        unsigned long long *bbox, const Counters &cnt, int *err, cudaStream_t st);
// Curve keys of all particles and their sorted order (keys_out, vals_out;
// keys_in and vals_in are scratch).  temp: sort_temp_bytes, unless the particles
// are few enough to sort in tiles.
bool sorts_in_tiles(int ntot);
size_t sort_temp_bytes(int ntot, int end_bit);
cudaError_t launch_sorted(const SetDesc *sets, int nsets, int max_n, int ntot, const InputsDev &in,
                          const unsigned long long *bbox, int bits, int end_bit, void *temp,
                          size_t temp_bytes, unsigned long long *keys_in, int *vals_in,
                          unsigned long long *keys_out, int *vals_out, cudaStream_t st);
// Sorted layout; resets bbox.  ilist non-null: also the row list of calls that
// compute every row of every set (otherwise launch_rows_range).
cudaError_t launch_gather(const SetDesc *sets, int nsets, int max_npad, const InputsDev &in,
                          const int *sorted_vals, SortedF64 D, SortedF32 F, int *ilist,
                          unsigned long long *bbox, cudaStream_t st);
// Row list of one set with rows [i_lo, i_lo + ni) selected in sorted order.
size_t select_temp_bytes(int n);
cudaError_t launch_rows_range(const SetDesc &set_host, const SortedF64 D, int *ilist,
                              int *nsel_dev, void *temp, size_t temp_bytes, cudaStream_t st);
// Records of META_J sorted slots, and (ntiles > 0) the i-tiles' centres.
cudaError_t launch_meta(const SetDesc *sets, int nmeta_total, const int *meta_set, int ntiles,
                        const int *tile_set, int itile, const int *ilist, const SortedF64 D,
                        JMeta *jmeta, ITileMeta *imeta, cudaStream_t st);

// --- compute kernels (sg_f64.cu, sg_f32.cu)
struct ComputeArgs {
    const SetDesc *sets;
    const WorkItem *items;
    int nitems;
    int *head;           // queue head, zeroed before the launch
    SortedF64 D;
    SortedF32 F;
    const int *ilist;
    const ITileMeta *imeta;
    const JMeta *jmeta;
    double *partials;    // [slot][4][itile], slot = WorkItem::slot
    // split-FP32: [slot][itile] sum over the item's j-tiles of |FP32 tile sum|^2
    // (acceleration components, both packed lanes): the scale of the FP32
    // rounding error of the row, merged into the refine test (nullable).
    // Negative: the row's near pairs are not in the item's sums (refine on)
    float *gpart;
    // when non-null the item count is read here instead of `nitems` (work
    // lists planned on the device, e.g. the FP64 refine of flagged rows)
    const int *nitems_dev;
    int *err;
    int nkernel;
    int itile;
    bool refine;         // split-FP32: listed rows are recomputed in FP64 (near pairs may be left to it)
    float band2;         // split-FP32: pairs with r^2 < band2 * max(H^2) use FP64 (>= 1)
    // split-FP32 built with -DSG_PHASES: [PHASE_COUNTERS] clock64 cycles per
    // phase summed over warps (see the Phase enum); nullptr = not counted
    unsigned long long *phases = nullptr;
};

// Phase accounting of the split-FP32 kernel (a diagnostic build: the pair
// kernel compiled with -DSG_PHASES).  Consumer and producer warps sum the
// SM cycles they spend in each phase; counts are per warp.
enum Phase {
    PH_ITEM = 0,      // consumer: waiting for the next item
    PH_ROWS,          // consumer: loading the item's rows, warp box
    PH_WAIT_FULL,     // consumer: waiting for a staged tile
    PH_FAR,           // consumer: far loop + tile fold
    PH_CHECKED,       // consumer: checked loop (near pairs masked) + tile fold
    PH_NEAR,          // consumer: near_eval (FP64 pairs)
    PH_END,           // consumer: combining and writing the item's partials
    PH_PROD_WAIT,     // producer: waiting for a free stage or for its copies
    PH_PROD_WORK,     // producer: issuing copies, rewriting tiles, tile boxes
    PH_N_FAR,         // count: far (warp, tile) pairs
    PH_N_CHECKED,     // count: checked (warp, tile) pairs
    PH_N_NEAR,        // count: near_eval calls
    PH_N_ITEMS,       // count: items started per consumer warp
    PHASE_COUNTERS = 16
};
bool phases_built();

struct VariantInfo {
    int precision;  // 0 fp64, 1 f32 split
    int nt;         // threads per block
    int k;          // rows per thread
    int q;          // threads per row
    int tj;         // j-tile
    int newton;     // one Newton step on rsqrt (f32 only)
    const char *name;
    int rows;       // rows per i-tile
    int itile() const { return rows; }
};
int variant_count(int precision);
const VariantInfo &variant_info(int precision, int v);
// Resident blocks per SM of variant v (queried once per process).
int variant_occupancy(int precision, int v);
cudaError_t launch_compute(int precision, int v, int grid, const ComputeArgs &a, cudaStream_t st);

// --- merge and diagnostics (sg_prep.cu)
// Refine test of the merge (split-FP32 calls): rows whose error scale G^2
// exceeds thresh2 * |a|^2, or whose near pairs were left out, are listed for the
// FP64 refine.
struct MergeRefine {
    const float *gpart = nullptr;  // [slot][itile] G^2 partials; null: no test
    double thresh2 = 0.0;          // T^2
    int *rcount = nullptr;         // [nsets] rows listed per set (zeroed before the merge)
    int *rlist = nullptr;          // listed sorted slots; set s at [S.ioff, S.ioff + S.ni)
    double *scale = nullptr;       // optional: G per row in the caller's order
};
// W of every set: the kernel that writes the tiles' sums lets its last block add
// them per set (count: its self-resetting block counter), or, from WSUM_SETS
// sets, leaves that to launch_wsum.
constexpr int WSUM_SETS = 256;
struct WSum {
    double *wtile = nullptr;    // per i-tile sums of m phi (null: no W)
    double *W = nullptr;
    unsigned *count = nullptr;  // zero between launches
    int nsets = 0;
};
// tile_slots[t] = (first partial slot, j-chunk count) of global i-tile t.
cudaError_t launch_merge(const SetDesc *sets, const int *tile_set, const int2 *tile_slots,
                         int ntiles_total, int itile, const int *ilist, const SortedF64 D,
                         const double *partials, OutputsDev out, const WSum &ws,
                         const MergeRefine &R, cudaStream_t st);
cudaError_t launch_wtile_out(const SetDesc *sets, const int *tile_set, int ntiles_total, int itile,
                             const int *ilist, const SortedF64 D, const double *pot, const WSum &ws,
                             cudaStream_t st);

// --- FP64 refine of the listed rows (sg_refine.cu)
// Plans the refine on the device from the per-set counts: for set s the rows
// rlist[S.ioff, S.ioff + rcount[s]) in tiles of `itile` rows, every tile
// split into the same number of j-chunks (enough items to fill `target`
// persistent blocks, at least 256 sources per chunk), one partial slot per
// item; sets with at most 32 listed rows take row-chunk items instead (one warp
// per row and source chunk), unless all of them together list more than
// REFINE_LIGHT_CAP rows.  Writes rsets (copies of sets with ni, ntiles, nchunks,
// slot_off of the refine), the items and their count.  At most max_items items
// are written; a plan that would need more sets DEVERR_INPUT (never expected:
// the host sizes max_items for every row flagged, in tiles).
// Row-chunk items that a refine plan may hold.
constexpr int REFINE_LIGHT_CAP = 65536;
cudaError_t launch_refine_plan(const SetDesc *sets, int nsets, const int *rcount, int itile,
                               int tj, int min_j, int target, int max_items, SetDesc *rsets,
                               WorkItem *items, int *nitems, int *nlight, int *nunits, int *err,
                               cudaStream_t st);
cudaError_t launch_refine_light(const SetDesc *rsets, int nsets, const int *nitems,
                                const int *rlist, const SortedF64 &D, int nkernel, double *lpart,
                                int sm_count, cudaStream_t st);
// Scatter the refined rows: chunk sums in a fixed order, written over the
// split-FP32 results in the caller's order; nunits counts the units of 32
// listed rows that the plan laid out (rsets' tile_off).
cudaError_t launch_refine_merge(const SetDesc *rsets, int nsets, const int *nunits, int itile_ref,
                                const int *rlist, const SortedF64 D, const double *rpart,
                                const double *lpart, OutputsDev out, int sm_count, cudaStream_t st);
cudaError_t launch_wsum(const SetDesc *sets, int nsets, const double *wtile, double *W,
                        cudaStream_t st);
cudaError_t launch_range2(int n, const double *hp, const double *u, double *range2, cudaStream_t st);
cudaError_t launch_kick(int n, double *x, double *y, double *z, double sigma,
                        unsigned long long seed, unsigned long long *counter, cudaStream_t st);
cudaError_t launch_fp32_probe(int iters, int blocks, float *sink, cudaStream_t st);
cudaError_t launch_fp64_probe(int iters, int blocks, float *sink, cudaStream_t st);
cudaError_t launch_wait_selftest(uint32_t polls, int *err, cudaStream_t st);

// --- Barnes-Hut octree (sg_tree.cu)
constexpr int TREE_LEAF = 16;    // a node with more particles splits
constexpr int TREE_LEVELS = 21;  // key bits per axis (one octree level per 3-bit digit)
// device level table: [L] first node of level L (L = 0..TREE_LEVELS + 1), then the
// node count the tree needs when the capacity does not suffice (else 0)
constexpr int TREE_LV_OVERFLOW = TREE_LEVELS + 2;
constexpr int TREE_LV_SIZE = TREE_LEVELS + 3;
constexpr int TREE_STACK = 8192; // traversal stack entries per warp
constexpr int TREE_GROUP = 32;   // particles of a walking group, at most
constexpr int TREE_BUDGET = 8192;  // particles within the largest H of a group's box (each
                                   // tested pair by pair) before the group is handed to the
                                   // direct FP64 sum; a typical group has ~500-800
constexpr int TREE_HEAVY_CHUNKS = 1024;  // most source chunks of a heavy group's direct sum
// Heavy groups a captured (device-counted) tree call can hand to the direct
// sum; more set DEVERR_TREE_CAP.  Partial sums: (4096 + cap) chunks.
constexpr int TREE_HEAVY_CAP = 4096;
// Source chunks per heavy group: about 4096 blocks in all, at least 256 sources
// each, 1..TREE_HEAVY_CHUNKS (n: the largest set's particles).  One heavy group of
// 40,961 particles: 20 chunks of 2,048 left most of the GPU idle for 142 us.
__host__ __device__ inline int tree_heavy_chunks(int nheavy, int n)
{
    int c = (4096 + nheavy - 1) / (nheavy > 0 ? nheavy : 1);
    if (c > n / 256) c = n / 256;
    return c < 1 ? 1 : (c > TREE_HEAVY_CHUNKS ? TREE_HEAVY_CHUNKS : c);
}

struct TreeNode {
    int start, end;     // sorted-slot range of its particles
    int child, nchild;  // first child (children are contiguous), count; 0: leaf
};
struct NodeGeom {      // bounding box and opening data (48 bytes)
    double cx, cy, cz; // box centre
    float hx, hy, hz;  // half sizes, rounded up
    float op2;         // (l / theta)^2, l = edge length
    float h2max;       // largest H^2 of its particles
    float pad_;
};
struct NodeMP {        // multipoles (64 bytes)
    double mx, my, mz; // centre of mass
    double m;          // mass
    float q[6];        // traceless quadrupole 3 S - tr(S) I about the centre of
                       // mass (S the second moment): xx yy zz xy xz yz
    float pad_[2];
};
struct TreeBuildArgs {
    int levels;                      // key digits per set: bits per axis (<= TREE_LEVELS)
    int nroots;                      // sets: level 0 holds one root per set
    int nslots, max_npad;            // sorted slots (pads included), of all sets and of the largest
    const SetDesc *sets;             // root s spans [sets[s].poff, sets[s].poff + sets[s].n)
    const unsigned long long *keys;  // sorted Hilbert keys, set s at [sets[s].off, + sets[s].n)
    TreeNode *nodes;
    int *parent, *done;              // per node: its parent (roots: -1), a zeroed counter
    int cap;                         // node capacity
    unsigned *bits;                  // scratch, tree_scan_items(nslots, levels) entries each
    int *cnt, *off;
    int *lv;                         // device level table (TREE_LV_SIZE ints)
    void *scan_temp;
    size_t scan_temp_bytes;
};
// One count per level >= 1 and 32 sorted slots, and a closing one for the total.
inline int tree_scan_items(int nslots, int levels) { return levels * (nslots / 32) + 1; }
// Parts a group's walk is cut into, by the particles of its set: one warp walks
// a group's nodes in sequence, so few groups leave most of the GPU idle and the
// longest walk sets the time.  From ~8,000 groups (~23 particles each) the walks
// of one set fill it; below, the count of (group, part) pairs is kept there, up
// to 8 parts (every part visits the nodes above level 3).
__host__ __device__ inline int tree_walk_parts(int n)
{
    int p = 1;
    while (p < 8 && (long long)n * p < 8000ll * 23) p *= 2;
    return p;
}
// The nodes whose particles are cut into walking groups hold at most this many.
// Longer runs fill more lanes (1M red giant: 41.1 ms with runs of siblings, 40.9
// with 128, 35.1 with 512, 33.6 with 2,048) but make fewer groups, which costs
// where the walks are too few to fill the GPU (40,961 particles: 1,617 us with
// 128, 1,645 with 512, 1,686 with 2,048): 128 for the sets whose walks are cut
// into parts.
__host__ __device__ inline int tree_group_node(int n) { return tree_walk_parts(n) > 1 ? 128 : 2048; }
struct TreeWalkArgs {
    const TreeNode *nodes;
    const NodeGeom *geom;
    const NodeMP *mp;
    SortedF64 D;
    int ngroups, nkernel;
    const int *ngroups_dev;    // when non-null the group count is read here
    int nroots;                // roots are nodes [0, nroots), one per set
    const SetDesc *sets;
    const int2 *groups;  // [ngroups] sorted-slot ranges (start, end), end - start <= 32
    int *head;       // group counter (zeroed before the launch)
    int *heavy;      // [ngroups] groups handed to the direct sum ...
    int *nheavy;     // ... and their count (zeroed before the launch)
    int *stack;      // TREE_STACK entries per walking warp
    int stack_cap;
    int nparts;      // most parts of any group's walk (tree_walk_parts)
    const int *parent;  // per node
    const int *lv;   // level table of the build
    int *gtaken;     // [ngroups] tested-list entries per group (zeroed before the launch)
    double *out;     // the sets' results (SetDesc::res_off), in sorted order
    int *err;
};
size_t tree_scan_temp_bytes(int n);
// Octree build without a host wait; t.lv receives the level table (nodes of level
// l are [lv[l], lv[l + 1])), all zero with the needed count in
// lv[TREE_LV_OVERFLOW] when `cap` nodes do not suffice (the caller regrows the
// node array and builds again).
cudaError_t tree_build(const TreeBuildArgs &t, cudaStream_t st);
// Counts that the host either knows (eager calls: read back) or leaves on the
// device (calls inside a graph capture): `dev` non-null means "read it there",
// `host` then bounds it (grids are sized for the bound, kernels loop).
struct DevCount {
    int host;
    const int *dev;
    __device__ int get() const { return dev ? *dev : host; }
};
// Lists the walking groups (order not significant); *ngroups via `count`.
cudaError_t tree_groups(DevCount nn, int nroots, const TreeNode *nodes, const int *parent,
                        int2 *glist, int *count, cudaStream_t st);
// Groups sorted by descending largest H^2 of their particles (walking order).
size_t tree_order_temp_bytes(int ng);
cudaError_t tree_order_groups(DevCount ng, const int2 *glist, int2 *ordered, const double *h2,
                              unsigned *keys_in, unsigned *keys_out, void *temp, size_t temp_bytes,
                              cudaStream_t st);
// Node properties, bottom-up; acc_buf: tree_acc_bytes(nn) of scratch.
size_t tree_acc_bytes(int nn);
cudaError_t tree_props(DevCount nn, const TreeNode *nodes, const int *parent, int *done,
                       const SortedF64 &D, double theta, void *acc_buf, NodeGeom *geom, NodeMP *mp,
                       int sm_count, cudaStream_t st);
int tree_walk_warps(int sm_count);
cudaError_t tree_walk(const TreeWalkArgs &a, int sm_count, cudaStream_t st);
// Slots of the sets' results: a set has as many parts as its own walk, however
// many the largest count in the batch is.
inline long long tree_res_slots(int n, int npad) { return (long long)npad * tree_walk_parts(n); }
// Where quantity q of part p of the set's sorted slot `slot` is in the results.
__host__ __device__ inline size_t tree_res_at(const SetDesc &S, int p, int q, int slot)
{
    return 4 * (size_t)S.res_off + ((size_t)p * 4 + q) * S.npad + (slot - S.poff);
}
// Rows [i_lo, i_lo + ni) to the caller's order, the parts added in order; W of
// every set (nullable) through wpart, nsets * tree_scatter_blocks(max_n) doubles.
int tree_scatter_blocks(int max_n);
cudaError_t tree_scatter(const SetDesc *sets, int nsets, int max_n, int i_lo, int ni,
                         const double *res, const SortedF64 &D, const OutputsDev &out,
                         double *wpart, double *W, cudaStream_t st);
// Direct FP64 sums over the group's own set for the groups the walk handed
// over (*nheavy on the device, at most `cap`; more set DEVERR_TREE_CAP).
// max_n: the largest set; nheavy_host > 0 sizes the grid exactly.
cudaError_t tree_heavy(int nheavy_host, const int *nheavy, int cap, const int *heavy,
                       const int2 *groups, const SetDesc *sets, const TreeNode *nodes, int nroots,
                       const SortedF64 &D, int max_n, int nkernel, double *partials, double *out,
                       int *err, cudaStream_t st);
// Partial-sum doubles tree_heavy needs for up to `cap` heavy groups.
size_t tree_heavy_partials(int cap, int max_n);
// Raises DEVERR_TREE_CAP when the build ran out of nodes (lv overflow flag).
cudaError_t tree_check_build(const int *lv, int *err, cudaStream_t st);

}  // namespace sg
