// sg_tree.cu -- Barnes-Hut octree gravity for sm_100a: the approximate
// alternative that the reference ships as a drop-in library with the same
// C-ABI (misc/SPHgravtree_lib: grav_force_tree.cu over libSequoia), written
// here from its semantics:
//   * an octree over the Hilbert-sorted particles (an octree cell is a
//     contiguous key range); a node splits while it holds more than
//     TREE_LEAF particles (the reference: 64);
//   * every node carries its mass, centre of mass and second moment about
//     it (monopole + quadrupole, as libSequoia's body_node), built bottom-up
//     in FP64; the walk uses the traceless quadrupole 3S - tr(S)I;
//   * particles are walked in groups of at most 32 along the curve
//     (k_tree_groups), one warp each, or up to eight for the groups of small
//     sets (tree_walk_parts), the groups
//     with the largest H first; a node is opened when the gap between the
//     group's and the node's bounding boxes is at most l / theta, l the
//     node's edge length (libSequoia's minimum-distance criterion,
//     compute_properties.cu:339, dev_shared_traverse_functions.cu:311-337);
//     theta comes from gpu_init_dev_ (main.f:269-270 passes 0.3).  It is
//     also opened when the gap is at most max(H) of the node's or the
//     group's particles, so every pair closer than the softening length is
//     evaluated particle by particle with the softened kernel (the reference
//     leaves that test out, INDSOFT); with theta -> 0 the walk is therefore
//     the direct sum;
//   * accepted nodes interact through the quadrupole expansion in FP32;
//     particles of opened leaves that lie farther than every H from the
//     group's box are Newtonian FP32 pairs without a per-pair test, the
//     others are tested pair by pair: FP32 when Newtonian, FP64 with the
//     CPU-path formulas (pair_f64_fast) for r < max(H_i, H_j) and r = 0;
//   * a group with more than TREE_BUDGET tested particles (a dense region
//     inside a softening sphere, e.g. a point-mass core with a large H)
//     leaves the walk and gets the direct FP64 sum over all particles
//     instead, spread over many CTAs (k_tree_heavy).
// Construction numbers all nodes with one prefix sum.  Atomics only order the
// group list, hand groups to warps and count a node's finished children; every
// sum has a fixed order, so the results are bit-for-bit reproducible.
#include "sg_launch.h"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>

namespace sg {

// ---------------------------------------------------------------- build
// The tree follows from the sorted keys position by position, without a pass
// per level.  Position k of a set starts a cell at every level from the one
// where its key first differs from position k - 1's; a cell of
// level L >= 1 is a node when its parent splits, i.e. when TREE_LEAF + 1
// consecutive positions around k share the first L - 1 digits.
// One warp handles 32 positions: it writes, per level, the bit mask and the
// count of the nodes that start there; one scan over (level, 32-position
// group), level by level, then numbers all nodes in level order, and every
// position writes its own nodes (end of the range by a galloping search, first
// child = its own node one level down, child count from the numbering).  Four
// launches for the whole tree, each bound by the latency of a few dependent
// loads.  Level by level (count, scan, bounds, emit, each thread searching its
// node's eight digits one after another) a 40,961-particle tree took 41
// launches and 510 us.
// Leading 3-bit digits that two keys of one set share.
__device__ __forceinline__ int common_digits(unsigned long long a, unsigned long long b, int levels)
{
    const unsigned long long x = a ^ b;
    return x == 0ull ? levels : min(levels, (3 * levels - 1 - (63 - __clzll(x))) / 3);
}

// Value at position index - o of a warp's 32 positions (hi) or the 32 before (lo).
__device__ __forceinline__ int back(int hi, int lo, int o, int lane)
{
    const int h = __shfl_up_sync(0xffffffffu, hi, o);
    const int l = __shfl_sync(0xffffffffu, lo, (lane + 32 - o) & 31);
    return lane >= o ? h : l;
}

__global__ void k_tree_bits(const SetDesc *sets, int nroots, int levels,
                            const unsigned long long *keys, int ngrp, unsigned *bits, int *cnt)
{
    static_assert(TREE_LEAF == 16, "the window maximum below is 17 positions wide");
    const int lane = threadIdx.x & 31;
    const int k0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) cnt[levels * ngrp] = 0;
    for (int set = blockIdx.y; set < nroots; set += gridDim.y) {
        const SetDesc S = sets[set];
        if (k0 >= S.npad) continue;
        const unsigned long long *key = keys + S.off;
        // shared digits of positions w and w + 16, for the warp's positions and the 16 before
        auto window = [&](int w) {
            return w >= 0 && w + TREE_LEAF < S.n ? common_digits(key[w], key[w + TREE_LEAF], levels) : -1;
        };
        int hi = window(k0 + lane), lo = window(k0 - 32 + lane);
#pragma unroll
        for (int o = 1; o <= 8; o <<= 1) {  // maximum over 2, 4, 8, 16 positions back
            const int h = back(hi, lo, o, lane);
            const int l = __shfl_up_sync(0xffffffffu, lo, o);
            hi = max(hi, h);
            if (lane >= o) lo = max(lo, l);
        }
        const int deepest = max(hi, back(hi, lo, 1, lane)) + 1;
        const int k = k0 + lane;
        int first = levels + 1;
        if (k < S.n) first = k == 0 ? 1 : common_digits(key[k - 1], key[k], levels) + 1;
        unsigned mine = 0u;
        for (int L = 1; L <= levels; L++) {
            const unsigned m = __ballot_sync(0xffffffffu, first <= L && L <= deepest);
            if (lane == L - 1) mine = m;
        }
        if (lane < levels) {
            const size_t g = (size_t)lane * ngrp + S.poff / 32 + k0 / 32;
            bits[g] = mine;
            cnt[g] = __popc(mine);
        }
    }
}

// Nodes [nroots, ...) from the numbering; level 0 holds one root per set over
// the set's sorted slots (its pads excluded).  lv[L] = first node of level L,
// lv[L + 1] its end (0 throughout when the node array is too small, so that
// nothing walks the tree; lv[TREE_LV_OVERFLOW] then holds the node count needed).
__global__ void k_tree_emit(const SetDesc *sets, int nroots, int levels,
                            const unsigned long long *keys, int ngrp, const unsigned *bits,
                            const int *off, int cap, TreeNode *nodes, int *parent, int *done,
                            int *lv)
{
    const int lane = threadIdx.x & 31;
    const long long total = (long long)nroots + off[levels * ngrp];
    const bool full = total > cap;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x <= TREE_LEVELS + 1) {
        const int L = threadIdx.x;
        int v = 0;
        if (!full && L > 0) v = nroots + off[min(L - 1, levels) * ngrp];
        lv[L] = v;
        if (L == 0) lv[TREE_LV_OVERFLOW] = full ? (int)min(total, 0x7fffffffll) : 0;
    }
    if (full) return;
    const int k0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32;
    for (int set = blockIdx.y; set < nroots; set += gridDim.y) {
        const SetDesc S = sets[set];
        if (k0 > 0 && k0 >= S.n) continue;
        const unsigned long long *key = keys + S.off;
        const int k = k0 + lane;
        const int g = S.poff / 32 + k0 / 32;
        const unsigned below = (1u << lane) - 1u;
        // nodes of level L that start before position p
        auto rank = [&](int L, int p) {
            const int q = S.poff + p, h = (L - 1) * ngrp + (q >> 5);
            int r = off[h];
            if (q & 31) r += __popc(bits[h] & ((1u << (q & 31)) - 1u));
            return nroots + r;
        };
        auto write = [&](int i, int start, int end, int L, int child) {
            TreeNode T;
            T.start = S.poff + start;
            T.end = S.poff + end;
            T.child = 0;
            T.nchild = 0;
            if (child >= 0) {
                T.child = child;
                T.nchild = rank(L + 1, end) - child;
                for (int c = 0; c < T.nchild; c++) parent[child + c] = i;
            }
            nodes[i] = T;
            done[i] = 0;
        };
        int child = -1;  // this position's node one level down
        int end = k + 1;
        for (int L = levels; L >= 1; L--) {
            const int h = (L - 1) * ngrp + g;
            const unsigned m = k0 < S.npad ? bits[h] : 0u;
            if (m == 0u) continue;
            if (!((m >> lane) & 1u)) {
                child = -1;
                continue;
            }
            // end of the cell: first position whose first L digits differ, by
            // galloping from the end of the cell one level down
            const int sh = 3 * (levels - L);
            const unsigned long long v = key[k] >> sh;
            int step = 1;
            while (end < S.n && (key[end] >> sh) == v) {
                end += step;
                step <<= 1;
            }
            if (step > 1) {  // the last probe that matched: end - step / 2
                int lo = end - (step >> 1) + 1, hi = min(end, S.n);
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if ((key[mid] >> sh) == v) lo = mid + 1;
                    else hi = mid;
                }
                end = lo;
            }
            const int i = nroots + off[h] + __popc(m & below);
            write(i, k, end, L, end - k > TREE_LEAF && L < levels ? child : -1);
            child = i;
        }
        if (k == 0) {
            parent[set] = -1;
            write(set, 0, S.n, 0, S.n > TREE_LEAF ? child : -1);
        }
    }
}

// Root (set) of a sorted slot: the last root starting at or before it.
// Roots are in set order; an empty set's root never holds a group.
__device__ __forceinline__ int root_of(const TreeNode *nodes, int nroots, int slot)
{
    int lo = 0, hi = nroots - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (nodes[mid].start <= slot) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Walking groups: the particles of every largest node with at most
// tree_group_node (a set's root, if small enough; a leaf of more coincident
// particles) in runs of even length, at most TREE_GROUP, along the curve; each
// particle lies in exactly one.  A warp walks a group, a particle per lane
// (runs of sibling nodes of at most 32 particles filled 23 lanes of
// 32 on the red giant).  Atomic order: results do not depend on which warp walks which group.
__global__ void k_tree_groups(DevCount nnc, int nroots, const TreeNode *nodes, const int *parent,
                              int2 *glist, int *count)
{
    const int nn = nnc.get();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const TreeNode T = nodes[i];
        const int n = T.end - T.start;
        const TreeNode R = nodes[nroots > 1 ? root_of(nodes, nroots, T.start) : 0];
        const int most = tree_group_node(R.end - R.start);
        if (n == 0 || (n > most && T.nchild > 0)) continue;
        const int p = parent[i];
        if (p >= 0) {
            const TreeNode U = nodes[p];
            if (U.end - U.start <= most) continue;  // the parent's groups hold it
        }
        const int g = (n + TREE_GROUP - 1) / TREE_GROUP;
        int k = atomicAdd(count, g);
        for (int c = 0; c < g; c++)
            glist[k++] = make_int2(T.start + (int)((long long)n * c / g),
                                   T.start + (int)((long long)n * (c + 1) / g));
    }
}

// ------------------------------------------------------------ properties
// Bottom-up in one launch: a warp sums a leaf's particles (fixed-order
// butterflies), and the warp that brings a node's last child goes on to that
// node, combining its children one per lane (masses and centres of mass
// combined, second moments moved to the new centre by the parallel-axis rule,
// in a fixed order whichever warp does it), all in FP64: reproducible.  Bound
// by the latency of the ~10 hand-overs from the deepest leaf to the root.  One
// launch per level, a thread looping over its node's children, took 98 us for
// a 40,961-particle tree.
struct NodeAcc {
    double m, c[3];   // mass, centre of mass
    double lo[3], hi[3];
    double s[6];      // second moment about c: xx yy zz xy xz yz
    double h2max;
};

template <int W>  // over aligned runs of W lanes
__device__ __forceinline__ double lanes_sum(double v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int W>
__device__ __forceinline__ double lanes_max(double v)
{
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Geometry and multipoles of a node for the walk.
__device__ __forceinline__ void finalize_node(const NodeAcc &A, double theta, NodeGeom *geom,
                                              NodeMP *mp)
{
    NodeGeom G;
    G.cx = 0.5 * (A.lo[0] + A.hi[0]);
    G.cy = 0.5 * (A.lo[1] + A.hi[1]);
    G.cz = 0.5 * (A.lo[2] + A.hi[2]);
    // half sizes rounded up by 2^-20 of the coordinates' magnitude, so
    // that float rounding never lets a node look farther than it is
    const double c3[3] = {G.cx, G.cy, G.cz};
    float hs[3];
    double hmax = 0.0;
    for (int d = 0; d < 3; d++) {
        const double h = 0.5 * (A.hi[d] - A.lo[d]);
        hs[d] = (float)(h + 9.5367e-7 * (fabs(c3[d]) + h));
        hmax = fmax(hmax, h);
    }
    G.hx = hs[0];
    G.hy = hs[1];
    G.hz = hs[2];
    const double l = 2.0 * hmax;  // edge length
    G.op2 = l > 0.0 ? (theta > 0.0 ? (float)((l / theta) * (l / theta)) : INFINITY) : 0.f;
    G.h2max = (float)A.h2max * 1.000001f;
    G.pad_ = 0.f;
    *geom = G;
    NodeMP P;
    P.mx = A.c[0];
    P.my = A.c[1];
    P.mz = A.c[2];
    P.m = A.m;
    // traceless quadrupole Q = 3 S - tr(S) I
    const double tr = A.s[0] + A.s[1] + A.s[2];
    P.q[0] = (float)(3.0 * A.s[0] - tr);
    P.q[1] = (float)(3.0 * A.s[1] - tr);
    P.q[2] = (float)(3.0 * A.s[2] - tr);
    for (int q = 3; q < 6; q++) P.q[q] = (float)(3.0 * A.s[q]);
    P.pad_[0] = P.pad_[1] = 0.f;
    *mp = P;
}

__global__ void __launch_bounds__(256) k_tree_props(DevCount nnc, const TreeNode *nodes,
                                                    const int *parent, int *done, SortedF64 D,
                                                    double theta, NodeAcc *acc, NodeGeom *geom,
                                                    NodeMP *mp)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int nn = nnc.get();
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int leaf = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); leaf < nn; leaf += nw) {
        const TreeNode T = nodes[leaf];
        if (T.nchild > 0) continue;
        double m = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
        NodeAcc A;
        A.h2max = 0.0;
        for (int d = 0; d < 3; d++) A.lo[d] = A.hi[d] = -INFINITY;  // lo: of -x
        for (int s = T.start + lane; s < T.end; s += 32) {
            const double w = D.m[s], x = D.x[s], y = D.y[s], z = D.z[s];
            m += w;
            mx += w * x;
            my += w * y;
            mz += w * z;
            A.h2max = fmax(A.h2max, D.h2[s]);
            A.lo[0] = fmax(A.lo[0], -x); A.lo[1] = fmax(A.lo[1], -y); A.lo[2] = fmax(A.lo[2], -z);
            A.hi[0] = fmax(A.hi[0], x);  A.hi[1] = fmax(A.hi[1], y);  A.hi[2] = fmax(A.hi[2], z);
        }
        A.m = lanes_sum<32>(m);
        mx = lanes_sum<32>(mx);
        my = lanes_sum<32>(my);
        mz = lanes_sum<32>(mz);
        A.h2max = lanes_max<32>(A.h2max);
        for (int d = 0; d < 3; d++) {
            A.lo[d] = -lanes_max<32>(A.lo[d]);
            A.hi[d] = lanes_max<32>(A.hi[d]);
        }
        // massless nodes sit at their box centre
        A.c[0] = A.m > 0.0 ? mx / A.m : 0.5 * (A.hi[0] + A.lo[0]);
        A.c[1] = A.m > 0.0 ? my / A.m : 0.5 * (A.hi[1] + A.lo[1]);
        A.c[2] = A.m > 0.0 ? mz / A.m : 0.5 * (A.hi[2] + A.lo[2]);
        for (int k = 0; k < 6; k++) A.s[k] = 0.0;
        for (int s = T.start + lane; s < T.end; s += 32) {
            const double w = D.m[s], x = D.x[s] - A.c[0], y = D.y[s] - A.c[1], z = D.z[s] - A.c[2];
            A.s[0] += w * x * x;
            A.s[1] += w * y * y;
            A.s[2] += w * z * z;
            A.s[3] += w * x * y;
            A.s[4] += w * x * z;
            A.s[5] += w * y * z;
        }
        for (int k = 0; k < 6; k++) A.s[k] = lanes_sum<32>(A.s[k]);
        for (int i = leaf;;) {
            const int p = parent[i];
            int last = 0;
            if (lane == 0) {
                finalize_node(A, theta, &geom[i], &mp[i]);
                if (p >= 0) {
                    acc[i] = A;
                    __threadfence();  // the sums before the count
                    last = atomicAdd(&done[p], 1) + 1 == nodes[p].nchild;
                    __threadfence();  // the count before the siblings' sums
                }
            }
            if (!__shfl_sync(FULL, last, 0)) break;  // the root, or a sibling is still missing
            __syncwarp();
            const TreeNode N = nodes[p];
            const bool has = lane < N.nchild;  // one child per lane, at most 8
            const double *c = (const double *)(acc + N.child + (has ? lane : 0));
            double v[sizeof(NodeAcc) / sizeof(double)];
#pragma unroll
            for (int k = 0; k < (int)(sizeof(v) / sizeof(double)); k++) v[k] = __ldcg(c + k);
            NodeAcc C;
            C.m = has ? v[0] : 0.0;
            for (int d = 0; d < 3; d++) {
                C.c[d] = v[1 + d];
                C.lo[d] = has ? v[4 + d] : INFINITY;
                C.hi[d] = has ? v[7 + d] : -INFINITY;
            }
            for (int k = 0; k < 6; k++) C.s[k] = has ? v[10 + k] : 0.0;
            C.h2max = has ? v[16] : 0.0;
            A.m = lanes_sum<8>(C.m);
            A.h2max = lanes_max<8>(C.h2max);
            for (int d = 0; d < 3; d++) {
                A.lo[d] = -lanes_max<8>(-C.lo[d]);
                A.hi[d] = lanes_max<8>(C.hi[d]);
                const double mc = lanes_sum<8>(C.m * C.c[d]);
                A.c[d] = A.m > 0.0 ? mc / A.m : 0.5 * (A.lo[d] + A.hi[d]);
            }
            const double dx = C.c[0] - A.c[0], dy = C.c[1] - A.c[1], dz = C.c[2] - A.c[2];
            A.s[0] = lanes_sum<8>(C.s[0] + C.m * dx * dx);
            A.s[1] = lanes_sum<8>(C.s[1] + C.m * dy * dy);
            A.s[2] = lanes_sum<8>(C.s[2] + C.m * dz * dz);
            A.s[3] = lanes_sum<8>(C.s[3] + C.m * dx * dy);
            A.s[4] = lanes_sum<8>(C.s[4] + C.m * dx * dz);
            A.s[5] = lanes_sum<8>(C.s[5] + C.m * dy * dz);
            i = p;
        }
    }
}

// -------------------------------------------------------------------- walk
constexpr int WALK_WARPS = 4;
constexpr int CELL_CAP = 64;  // < 32 pending + 32 appended per step
constexpr int PART_CAP = 64;
constexpr int CELL_REC = 10;  // packed pairs of an accepted-node record

// Softened (or r = 0) pair of two sorted slots, out of the walk's way.
__device__ __noinline__ PairOut pair_of_slots(const SortedF64 &D, int nkernel, int si, int j)
{
    return pair_f64_fast(D, nkernel, si, j, D.x[j] - D.x[si], D.y[j] - D.y[si], D.z[j] - D.z[si],
                         D.m[j], D.h2[si], D.h2[j]);
}

// SPLIT: a group's walk is cut into parts (tree_walk_parts), one warp each.
template <bool SPLIT>
__global__ void __launch_bounds__(WALK_WARPS * 32, 5) k_tree_walk(const __grid_constant__ TreeWalkArgs a)
{
    // accepted nodes, group-relative, two to a record of CELL_REC packed pairs
    // {x y z M Qxx Qyy Qzz Qxy Qxz Qyz}
    __shared__ __align__(16) float s_cell[WALK_WARPS][CELL_CAP / 2 * CELL_REC * 2];
    // particles farther than any H from the whole group, two to a record {x y z m}
    __shared__ __align__(16) float s_far[WALK_WARPS][PART_CAP / 2 * 8];
    // the other particles: x y z m H^2 and their sorted slot
    __shared__ float s_part[WALK_WARPS][5][PART_CAP];
    __shared__ int s_pslot[WALK_WARPS][PART_CAP];
    __shared__ int s_q[WALK_WARPS][64];           // FP64 pairs: owner lane << 8 | entry
    __shared__ double s_qres[WALK_WARPS][4][32];  // their results
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    int *stack = a.stack + (size_t)(blockIdx.x * WALK_WARPS + w) * a.stack_cap;
    const SortedF64 D = a.D;
    float *cl = s_cell[w];
    float *fl = s_far[w];
    float(*pl)[PART_CAP] = s_part[w];
    int *ps = s_pslot[w];
    int *q = s_q[w];
    double(*qr)[32] = s_qres[w];
    const int ngroups = a.ngroups_dev ? *a.ngroups_dev : a.ngroups;

    const int level3 = SPLIT ? a.lv[3] : 0;

    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.head, 1);
        item = __shfl_sync(FULL, item, 0);
        const int g = SPLIT ? item / a.nparts : item, part = SPLIT ? item - g * a.nparts : 0;
        if (g >= ngroups) break;
        const int2 grp = a.groups[g];
        const int root = a.nroots > 1 ? root_of(a.nodes, a.nroots, grp.x) : 0;
        // The level-3 nodes, with all below them, are dealt out to the parts
        // by the sum of their and their ancestors' places among their
        // siblings; the nodes above are walked by every part, their own terms
        // dealt out alike.  All of it is the set's own, so a set's sums are
        // the same in a batch and alone.
        int P = 1, rchild = 0;
        if (SPLIT) {
            const TreeNode R = a.nodes[root];
            rchild = R.child;
            P = tree_walk_parts(R.end - R.start);
            if (part >= P) continue;
        }
        const int s0 = grp.x;
        const int s = s0 + lane;
        const bool act = s < grp.y;
        const int sr = act ? s : s0;  // inactive lanes mirror the group's first particle
        const double px = D.x[sr], py = D.y[sr], pz = D.z[sr];
        double lo[3] = {px, py, pz}, hi[3] = {px, py, pz};
        float gh2 = act ? (float)D.h2[s] : 0.f;
        for (int o = 16; o > 0; o >>= 1) {
            for (int d = 0; d < 3; d++) {
                lo[d] = fmin(lo[d], __shfl_xor_sync(FULL, lo[d], o));
                hi[d] = fmax(hi[d], __shfl_xor_sync(FULL, hi[d], o));
            }
            gh2 = fmaxf(gh2, __shfl_xor_sync(FULL, gh2, o));
        }
        gh2 *= 1.000001f;
        const double cx = 0.5 * (lo[0] + hi[0]), cy = 0.5 * (lo[1] + hi[1]),
                     cz = 0.5 * (lo[2] + hi[2]);
        const float ghx = (float)(0.5 * (hi[0] - lo[0]) * (1.0 + 1e-6) + 1e-30);
        const float ghy = (float)(0.5 * (hi[1] - lo[1]) * (1.0 + 1e-6) + 1e-30);
        const float ghz = (float)(0.5 * (hi[2] - lo[2]) * (1.0 + 1e-6) + 1e-30);
        const float xi = (float)(px - cx), yi = (float)(py - cy), zi = (float)(pz - cz);
        const f2 xi2 = pk(xi, xi), yi2 = pk(yi, yi), zi2 = pk(zi, zi);
        const float h2i = act ? (float)D.h2[s] : 0.f;
        // sums: each list flush in FP32, flushes and FP64 near pairs in FP64
        double fx = 0.0, fy = 0.0, fz = 0.0, fp = 0.0;
        int ncell = 0, nfar = 0, npart = 0, top = 1;
        int taken = 0;  // tested-list entries not yet reported to the group's count
        bool overflow = false, heavy = false;
        // Adds this part's entries to the group's count; whichever addition
        // passes TREE_BUDGET hands the group over, and every later one stops:
        // the total alone decides, not the order.
        auto report = [&]() {
            if (!SPLIT) {
                if (taken <= TREE_BUDGET) return false;
                if (lane == 0) a.heavy[atomicAdd(a.nheavy, 1)] = g;
                taken = 0;
                return true;
            }
            int over = 0;
            if (lane == 0 && taken > 0) {
                const int old = atomicAdd(&a.gtaken[g], taken);
                over = old + taken > TREE_BUDGET;
                if (over && old <= TREE_BUDGET) a.heavy[atomicAdd(a.nheavy, 1)] = g;
            }
            taken = 0;
            return __shfl_sync(FULL, over, 0) != 0;
        };
        // the walk starts at the root of the group's own set
        if (lane == 0) stack[0] = root;
        __syncwarp();

        // Every accepted node's box is disjoint from the group's (its gap is
        // above zero), so r > 0 for every lane, the idle ones included (they
        // mirror a particle of the group): no lane needs a guard.
        //   a = M d/r^3 - Q d/r^5 + 2.5 (d.Q.d) d/r^7,  phi = -M/r - 0.5 (d.Q.d)/r^5
        // in packed f32x2 arithmetic, two nodes per instruction: with
        // t = (d.Q.d)/r^4 the terms are d (M + 2.5 t)/r^3 - Q d/r^5 and
        // (M + 0.5 t)/r, 33 FMA-pipe instructions and 2 MUFU for two nodes.
        auto eval_cells = [&]() {
            if (ncell & 1) {  // an odd last node pairs with a massless copy of itself
                const float *c = cl + (ncell >> 1) * (2 * CELL_REC);
                if (lane < CELL_REC)
                    cl[(ncell >> 1) * (2 * CELL_REC) + 2 * lane + 1] = lane < 3 ? c[2 * lane] : 0.f;
                __syncwarp();
            }
            f2 ax = 0ull, ay = 0ull, az = 0ull, pp = 0ull;
            const f2 k25 = pk(2.5f, 2.5f), k05 = pk(0.5f, 0.5f);
#pragma unroll 2
            for (int e = 0; e < ncell; e += 2) {
                const ulonglong2 *c = (const ulonglong2 *)(cl + (e >> 1) * (2 * CELL_REC));
                const ulonglong2 A = c[0], B = c[1], C = c[2], E = c[3], G = c[4];
                const f2 dx = sub2(A.x, xi2), dy = sub2(A.y, yi2), dz = sub2(B.x, zi2);
                const f2 r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
                float ra, rb;
                upk(r2, ra, rb);
                const f2 ri = pk(rsqrt_approx(ra), rsqrt_approx(rb));
                const f2 ri2 = mul2(ri, ri), ri3 = mul2(ri2, ri), ri4 = mul2(ri2, ri2);
                // Q d: M = B.y, Qxx = C.x, Qyy = C.y, Qzz = E.x, Qxy = E.y, Qxz = G.x, Qyz = G.y
                const f2 qx = fma2(G.x, dz, fma2(E.y, dy, mul2(C.x, dx)));
                const f2 qy = fma2(G.y, dz, fma2(C.y, dy, mul2(E.y, dx)));
                const f2 qz = fma2(E.x, dz, fma2(G.y, dy, mul2(G.x, dx)));
                const f2 t = mul2(fma2(dz, qz, fma2(dy, qy, mul2(dx, qx))), ri4);
                const f2 f = mul2(fma2(k25, t, B.y), ri3), h = mul2(ri3, ri2);
                ax = sub2(fma2(f, dx, ax), mul2(h, qx));
                ay = sub2(fma2(f, dy, ay), mul2(h, qy));
                az = sub2(fma2(f, dz, az), mul2(h, qz));
                pp = fma2(ri, fma2(k05, t, B.y), pp);
            }
            float a, b;
            upk(ax, a, b);
            fx += (double)(a + b);
            upk(ay, a, b);
            fy += (double)(a + b);
            upk(az, a, b);
            fz += (double)(a + b);
            upk(pp, a, b);
            fp -= (double)(a + b);
            ncell = 0;
            __syncwarp();
        };
        // Far particles: Newtonian FP32 pairs, no per-pair test (r > 0 as
        // above), two sources per packed instruction.
        auto eval_far = [&]() {
            if (nfar & 1) {
                const float *c = fl + (nfar >> 1) * 8;
                if (lane < 4) fl[(nfar >> 1) * 8 + 2 * lane + 1] = lane < 3 ? c[2 * lane] : 0.f;
                __syncwarp();
            }
            f2 ax = 0ull, ay = 0ull, az = 0ull, pot = 0ull;
#pragma unroll 2
            for (int e = 0; e < nfar; e += 2) {
                const ulonglong2 *c = (const ulonglong2 *)(fl + (e >> 1) * 8);
                const ulonglong2 A = c[0], B = c[1];
                const f2 dx = sub2(A.x, xi2), dy = sub2(A.y, yi2), dz = sub2(B.x, zi2);
                const f2 r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
                float ra, rb;
                upk(r2, ra, rb);
                const f2 ri = pk(rsqrt_approx(ra), rsqrt_approx(rb));
                const f2 mr = mul2(B.y, ri), mr3 = mul2(mr, mul2(ri, ri));
                ax = fma2(mr3, dx, ax);
                ay = fma2(mr3, dy, ay);
                az = fma2(mr3, dz, az);
                pot = add2(pot, mr);
            }
            float a, b;
            upk(ax, a, b);
            fx += (double)(a + b);
            upk(ay, a, b);
            fy += (double)(a + b);
            upk(az, a, b);
            fz += (double)(a + b);
            upk(pot, a, b);
            fp -= (double)(a + b);
            nfar = 0;
            __syncwarp();
        };
        // Particles that may lie within some H of some lane: tested per pair;
        // softened (or r = 0) pairs are queued as (owner lane, list entry) and
        // evaluated in FP64 one per lane, 32 at a time, each owner adding its
        // own results in queue order.
        auto eval_parts = [&]() {
            float ax = 0.f, ay = 0.f, az = 0.f, pot = 0.f;
            int nq = 0;
            for (int e = 0; e <= npart; e++) {  // the last step empties the queue
                if (e < npart) {
                    const float dx = pl[0][e] - xi, dy = pl[1][e] - yi, dz = pl[2][e] - zi;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    const bool near = act && !(r2 >= fmaxf(h2i, pl[4][e]));
                    if (act && !near) {
                        const float ri = rsqrt_approx(r2);
                        const float mr = pl[3][e] * ri;
                        const float mr3 = mr * ri * ri;
                        ax += mr3 * dx;
                        ay += mr3 * dy;
                        az += mr3 * dz;
                        pot -= mr;
                    }
                    const unsigned nm = __ballot_sync(FULL, near);
                    if (near) q[nq + __popc(nm & below)] = (lane << 8) | e;
                    nq += __popc(nm);
                    __syncwarp();
                }
                if (nq < 32 && (e < npart || nq == 0)) continue;
                const int cnt = min(nq, 32);
                if (lane < cnt) {
                    const int o = q[lane] >> 8;
                    const PairOut r = pair_of_slots(a.D, a.nkernel, s0 + o, ps[q[lane] & 255]);
                    qr[0][lane] = r.ax;
                    qr[1][lane] = r.ay;
                    qr[2][lane] = r.az;
                    qr[3][lane] = r.pot;
                }
                __syncwarp();
                for (int t = 0; t < cnt; t++) {
                    if ((q[t] >> 8) == lane) {
                        fx += qr[0][t];
                        fy += qr[1][t];
                        fz += qr[2][t];
                        fp += qr[3][t];
                    }
                }
                __syncwarp();
                const int rest = nq - cnt;  // < 32: move them to the front
                const int v = lane < rest ? q[32 + lane] : 0;
                __syncwarp();
                if (lane < rest) q[lane] = v;
                nq = rest;
                __syncwarp();
            }
            fx += ax;
            fy += ay;
            fz += az;
            fp += pot;
            npart = 0;
            __syncwarp();
        };

        // One site for each list's evaluation, the last pass over an empty stack
        // included: inlined twice they made the kernel outgrow the instruction
        // cache (41% of the stalls were instruction fetches).
        for (bool more = true; more;) {
            more = top > 0;
            const int flush = more ? 32 : 1;  // entries that a list is evaluated from
            const int nb = min(top, 32);
            top -= nb;
            const int node = lane < nb ? stack[top + lane] : -1;
            __syncwarp();  // popped before the pushes below overwrite the slots
            bool cell = false;
            int nch = 0, ch0 = 0, chs = 1;  // children pushed: ch0, ch0 + chs, ...
            int lbeg = 0, lcnt = 0;         // an opened leaf's particles
            if (node >= 0) {
                const NodeGeom G = a.geom[node];
                const float gx = fmaxf(0.f, (float)fabs(G.cx - cx) - (G.hx + ghx));
                const float gy = fmaxf(0.f, (float)fabs(G.cy - cy) - (G.hy + ghy));
                const float gz = fmaxf(0.f, (float)fabs(G.cz - cz) - (G.hz + ghz));
                const float d2 = gx * gx + gy * gy + gz * gz;
                const bool open = d2 <= G.op2 || d2 <= fmaxf(G.h2max, gh2);
                const TreeNode T = a.nodes[node];
                bool mine = true, deal = false;
                int place = 0;
                if (SPLIT && P > 1 && node < level3) {
                    if (node != root) {
                        const int q = a.parent[node];
                        place = node - (q == root ? rchild : a.nodes[q].child);
                        if (q != root) {
                            place += q - rchild;
                            deal = true;  // a level-2 node: its children are dealt out
                        }
                    }
                    mine = place % P == part;
                }
                cell = !open && mine;
                if (open) {
                    if (T.nchild > 0) {
                        nch = T.nchild;
                        ch0 = T.child;
                        if (deal) {
                            const int skip = (part + P - place % P) % P;
                            ch0 += skip;
                            nch = nch > skip ? (nch - skip + P - 1) / P : 0;
                            chs = P;
                        }
                    } else if (mine) {
                        lbeg = T.start;
                        lcnt = T.end - T.start;
                    }
                }
            }
            // accepted nodes join the cell list (group-relative coordinates)
            const unsigned cm = __ballot_sync(FULL, cell);
            if (cell) {
                const int p = ncell + __popc(cm & below);
                const NodeMP P = a.mp[node];
                float *c = cl + (p >> 1) * (2 * CELL_REC) + (p & 1);
                c[0] = (float)(P.mx - cx);
                c[2] = (float)(P.my - cy);
                c[4] = (float)(P.mz - cz);
                c[6] = (float)P.m;
#pragma unroll
                for (int k = 0; k < 6; k++) c[8 + 2 * k] = P.q[k];
            }
            ncell += __popc(cm);
            __syncwarp();
            if (ncell >= flush) eval_cells();
            // opened inner nodes push their children
            const int incl = warp_inclusive(nch, lane);
            const int pushed = __shfl_sync(FULL, incl, 31);
            if (top + pushed > a.stack_cap) {
                overflow = true;  // reported below; the group's sums are not complete
                break;
            }
            for (int c = 0; c < nch; c++) stack[top + incl - nch + c] = ch0 + c * (SPLIT ? chs : 1);
            top += pushed;
            __syncwarp();
            // The particles of all opened leaves of the batch, one after another,
            // 32 to a step, join the far list or the tested list (leaf by leaf,
            // a step held ~10 of them and waited for the leaf's bounds first).
            const int linc = warp_inclusive(lcnt, lane);
            const int ltot = __shfl_sync(FULL, linc, 31);
            for (int b = 0; b < max(ltot, more ? 0 : 1); b += 32) {
                const int k = b + lane;
                const int ow = warp_owner(linc, k);
                const int j = __shfl_sync(FULL, lbeg - (linc - lcnt), ow) + k;
                const bool has = k < ltot;
                bool far = false;
                float ex = 0.f, ey = 0.f, ez = 0.f, em = 0.f, eh2 = 0.f;
                if (has) {
                    ex = (float)(D.x[j] - cx);
                    ey = (float)(D.y[j] - cy);
                    ez = (float)(D.z[j] - cz);
                    em = (float)D.m[j];
                    eh2 = (float)D.h2[j] * 1.000001f;
                    // a lower bound of the particle's distance to the group's
                    // box (1e-6 covers the FP32 roundings of ex and this sum)
                    const float bx = fmaxf(0.f, fabsf(ex) * (1.f - 1e-6f) - ghx);
                    const float by = fmaxf(0.f, fabsf(ey) * (1.f - 1e-6f) - ghy);
                    const float bz = fmaxf(0.f, fabsf(ez) * (1.f - 1e-6f) - ghz);
                    far = (bx * bx + by * by + bz * bz) * 0.9999f > fmaxf(eh2, gh2);
                }
                const unsigned fm = __ballot_sync(FULL, has && far);
                const unsigned tm = __ballot_sync(FULL, has && !far);
                if (has && far) {
                    const int p = nfar + __popc(fm & below);
                    float *c = fl + (p >> 1) * 8 + (p & 1);
                    c[0] = ex;
                    c[2] = ey;
                    c[4] = ez;
                    c[6] = em;
                }
                if (has && !far) {
                    const int p = npart + __popc(tm & below);
                    pl[0][p] = ex;
                    pl[1][p] = ey;
                    pl[2][p] = ez;
                    pl[3][p] = em;
                    pl[4][p] = eh2;
                    ps[p] = j;
                }
                nfar += __popc(fm);
                npart += __popc(tm);
                taken += __popc(tm);
                __syncwarp();
                if ((!SPLIT || taken >= 256) && report()) {
                    heavy = true;  // the group goes to the direct sum
                    break;
                }
                if (nfar >= flush) eval_far();
                if (npart >= flush) eval_parts();
            }
            if (heavy) break;
        }
        if (heavy || report()) continue;
        if (overflow && lane == 0) atomicOr(a.err, DEVERR_TREE);
        if (act) {
            const SetDesc S = a.sets[root];
            double *o = a.out + tree_res_at(S, part, 0, s);
            o[0] = fx;
            o[(size_t)S.npad] = fy;
            o[2 * (size_t)S.npad] = fz;
            o[3 * (size_t)S.npad] = fp;
        }
    }
}

// Direct FP64 sum of a heavy group: block (h, c) sums the group's <= 32
// particles (lane = row) over source chunk c (the block's warps take
// interleaved sources); warps combine in order, chunks merge in order.
constexpr int HEAVY_WARPS = 8;
// Block b works on (heavy group, source chunk) pairs b, b + grid, ...: chunk c
// of the group's own set, one row per lane, sources split over the warps.
// The chunk count follows the number of heavy groups (read on the device).
__global__ void __launch_bounds__(HEAVY_WARPS * 32)
k_tree_heavy(const int *nheavy_p, int cap, const int *heavy, const int2 *groups,
             const TreeNode *nodes, int nroots, SortedF64 D, int max_n, int nkernel,
             double *partials, int *err)
{
    __shared__ double sh[HEAVY_WARPS][4][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nh_all = *nheavy_p;
    if (nh_all > cap && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, DEVERR_TREE_CAP);
    const int nheavy = min(nh_all, cap);
    const int nchunks = tree_heavy_chunks(nheavy, max_n);
    for (int b = blockIdx.x; b < nheavy * nchunks; b += gridDim.x) {
        const int h = b / nchunks, c = b % nchunks;
        const int2 grp = groups[heavy[h]];
        const TreeNode R = nodes[nroots > 1 ? root_of(nodes, nroots, grp.x) : 0];
        const int ns = R.end - R.start;
        const int si = grp.x + lane;
        const bool act = si < grp.y;
        const int jb = R.start + (int)((long long)ns * c / nchunks);
        const int je = R.start + (int)((long long)ns * (c + 1) / nchunks);
        double sx = 0.0, sy = 0.0, sz = 0.0, sp = 0.0;
        if (act) {
            const double xi = D.x[si], yi = D.y[si], zi = D.z[si], h2i = D.h2[si];
            for (int j = jb + w; j < je; j += HEAVY_WARPS) {
                const PairOut o = pair_f64_fast(D, nkernel, si, j, D.x[j] - xi, D.y[j] - yi,
                                                D.z[j] - zi, D.m[j], h2i, D.h2[j]);
                sx += o.ax;
                sy += o.ay;
                sz += o.az;
                sp += o.pot;
            }
        }
        __syncthreads();  // the previous pair's reduction has read sh
        sh[w][0][lane] = sx;
        sh[w][1][lane] = sy;
        sh[w][2][lane] = sz;
        sh[w][3][lane] = sp;
        __syncthreads();
        if (w == 0) {
            for (int q = 0; q < 4; q++) {
                double v = sh[0][q][lane];
                for (int k = 1; k < HEAVY_WARPS; k++) v += sh[k][q][lane];
                partials[(((size_t)h * nchunks + c) * 4 + q) * 32 + lane] = v;
            }
        }
    }
}

// A block per heavy group h: warp (q, s) sums quantity q of chunks s, s + 8, ... in
// order, then the eight sums add in order.
constexpr int HEAVY_MERGE_SLICES = 8;
__global__ void __launch_bounds__(4 * HEAVY_MERGE_SLICES * 32)
k_tree_heavy_merge(const int *nheavy_p, int cap, const int *heavy,
                   const int2 *groups, const SetDesc *sets, const TreeNode *nodes, int nroots,
                   int max_n, const double *partials, double *out)
{
    __shared__ double s_sum[HEAVY_MERGE_SLICES][4][32];
    const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 3, slice = threadIdx.x >> 7;
    const int nheavy = min(*nheavy_p, cap);
    const int nchunks = tree_heavy_chunks(nheavy, max_n);
    for (int h = blockIdx.x; h < nheavy; h += gridDim.x) {
        const int2 grp = groups[heavy[h]];
        const int si = grp.x + lane;
        double v = 0.0;
#pragma unroll 4
        for (int c = slice; c < nchunks; c += HEAVY_MERGE_SLICES)
            v += partials[(((size_t)h * nchunks + c) * 4 + q) * 32 + lane];
        __syncthreads();  // the previous group's sums have been read
        s_sum[slice][q][lane] = v;
        __syncthreads();
        if (slice != 0 || si >= grp.y) continue;
        for (int k = 1; k < HEAVY_MERGE_SLICES; k++) v += s_sum[k][q][lane];
        const SetDesc S = sets[nroots > 1 ? root_of(nodes, nroots, grp.x) : 0];
        out[tree_res_at(S, 0, q, si)] = v;
        for (int p = 1; p < tree_walk_parts(S.n); p++) out[tree_res_at(S, p, q, si)] = 0.0;
    }
}

size_t tree_heavy_partials(int cap, int max_n)
{
    // nheavy * tree_heavy_chunks(nheavy, .) <= 4096 + nheavy for every nheavy <= cap
    (void)max_n;
    return ((size_t)4096 + (size_t)cap) * 4 * 32;
}

cudaError_t tree_heavy(int nheavy_host, const int *nheavy, int cap, const int *heavy,
                       const int2 *groups, const SetDesc *sets, const TreeNode *nodes, int nroots,
                       const SortedF64 &D, int max_n, int nkernel, double *partials, double *out,
                       int *err, cudaStream_t st)
{
    // eager calls know the count: one block per (group, chunk); captured
    // calls size the grid for the most chunks any count can give
    const int blocks = nheavy_host > 0
                           ? std::min(nheavy_host, cap) * tree_heavy_chunks(std::min(nheavy_host, cap), max_n)
                           : 4096;
    k_tree_heavy<<<blocks, HEAVY_WARPS * 32, 0, st>>>(nheavy, cap, heavy, groups, nodes, nroots, D,
                                                     max_n, nkernel, partials, err);
    ++g_launches;
    const int mblocks = nheavy_host > 0 ? std::min(nheavy_host, cap) : 256;
    k_tree_heavy_merge<<<mblocks, 4 * HEAVY_MERGE_SLICES * 32, 0, st>>>(
        nheavy, cap, heavy, groups, sets, nodes, nroots, max_n, partials, out);
    ++g_launches;
    return cudaGetLastError();
}

// Sorted-order results to the caller's rows [i_lo, i_lo + ni): the parts of a
// group's walk add in order; block (b, set) also sums m phi over its share of
// the set's slots (a contiguous run, in a fixed order) for W.
constexpr int SCATTER_NT = 256;
__global__ void __launch_bounds__(SCATTER_NT)
k_tree_scatter(const SetDesc *sets, int nsets, int i_lo, int ni, const double *res,
               SortedF64 D, OutputsDev out, double *wpart)
{
    __shared__ double s_w[SCATTER_NT];
    for (int set = blockIdx.y; set < nsets; set += gridDim.y) {
        const SetDesc S = sets[set];
        const int nparts = tree_walk_parts(S.n);
        const int per = ((S.n + gridDim.x - 1) / gridDim.x + SCATTER_NT - 1) / SCATTER_NT * SCATTER_NT;
        const int k0 = min(S.n, (int)min((long long)S.n, (long long)blockIdx.x * per));
        const int k1 = min(S.n, k0 + per);
        double w = 0.0;
        for (int k = k0 + threadIdx.x; k < k1; k += SCATTER_NT) {
            const int s = S.poff + k;
            double v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = res[tree_res_at(S, 0, q, s)];
            for (int p = 1; p < nparts; p++) {
#pragma unroll
                for (int q = 0; q < 4; q++) v[q] += res[tree_res_at(S, p, q, s)];
            }
            w += D.m[s] * v[3];
            const int o = D.orig[s];
            if (o < i_lo || o >= i_lo + ni) continue;
            out.ax[o] = v[0];
            out.ay[o] = v[1];
            out.az[o] = v[2];
            out.pot[o] = v[3];
        }
        if (!wpart) continue;
        __syncthreads();  // the previous set's sum has been read
        s_w[threadIdx.x] = w;
        __syncthreads();
        for (int o = SCATTER_NT / 2; o > 0; o >>= 1) {
            if ((int)threadIdx.x < o) s_w[threadIdx.x] += s_w[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) wpart[(size_t)set * gridDim.x + blockIdx.x] = s_w[0];
    }
}

// W = 1/2 sum m phi of every set from its blocks' sums: one block per set, fixed order.
__global__ void __launch_bounds__(SCATTER_NT) k_tree_wsum(int nblocks, const double *wpart, double *W)
{
    __shared__ double s_w[SCATTER_NT];
    double w = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += SCATTER_NT) w += wpart[(size_t)blockIdx.x * nblocks + b];
    s_w[threadIdx.x] = w;
    __syncthreads();
    for (int o = SCATTER_NT / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) s_w[threadIdx.x] += s_w[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) W[blockIdx.x] = 0.5 * s_w[0];
}

__global__ void k_tree_check_build(const int *lv, int *err)
{
    if (lv[TREE_LV_OVERFLOW]) atomicOr(err, DEVERR_TREE_CAP);
}

cudaError_t tree_check_build(const int *lv, int *err, cudaStream_t st)
{
    k_tree_check_build<<<1, 1, 0, st>>>(lv, err);
    ++g_launches;
    return cudaGetLastError();
}

// --------------------------------------------------------------- driver
size_t tree_scan_temp_bytes(int n)
{
    size_t b = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, b, (const int *)nullptr, (int *)nullptr, std::max(n, 1));
    return b;
}

cudaError_t tree_build(const TreeBuildArgs &t, cudaStream_t st)
{
    const int ngrp = t.nslots / 32;
    const dim3 grid((t.max_npad / 32 + 7) / 8, grid_sets(t.nroots));
    if (ngrp > 0) {
        k_tree_bits<<<grid, 256, 0, st>>>(t.sets, t.nroots, t.levels, t.keys, ngrp, t.bits, t.cnt);
        ++g_launches;
        size_t tb = t.scan_temp_bytes;
        const cudaError_t e = cub::DeviceScan::ExclusiveSum(t.scan_temp, tb, t.cnt, t.off,
                                                            tree_scan_items(t.nslots, t.levels), st);
        if (e != cudaSuccess) return e;
        ++g_launches;
    }
    k_tree_emit<<<grid, 256, 0, st>>>(t.sets, t.nroots, t.levels, t.keys, ngrp, t.bits, t.off, t.cap,
                                      t.nodes, t.parent, t.done, t.lv);
    ++g_launches;
    return cudaGetLastError();
}

static int grid_for(DevCount c, int per_block, int cap_blocks)
{
    return std::max(1, std::min((std::max(c.host, 1) + per_block - 1) / per_block, cap_blocks));
}

cudaError_t tree_groups(DevCount nn, int nroots, const TreeNode *nodes, const int *parent,
                        int2 *glist, int *count, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    k_tree_groups<<<grid_for(nn, 256, 4096), 256, 0, st>>>(nn, nroots, nodes, parent, glist, count);
    ++g_launches;
    return cudaGetLastError();
}

// Walking order: the largest H first.  Every particle within H of a group
// is tested pair by pair, so those groups walk longest; started first, they
// do not leave one warp running after the rest (results do not depend on the
// order: each group's sums are its own).  Entries past the group count (a
// device count bounded by ng.host) have key 0 and sort last.
__global__ void k_tree_group_keys(DevCount ngc, int bound, const int2 *glist, const double *h2,
                                  unsigned *keys)
{
    const int ng = ngc.get();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= bound) return;
    double m = 0.0;
    if (g < ng) {
        const int2 r = glist[g];
        for (int s = r.x; s < r.y; s++) m = fmax(m, h2[s]);
    }
    // non-negative floats order as their bits, the exponents alone sorted; a
    // group whose H^2 has none (a subnormal float) ties with the unused entries,
    // which the stable sort leaves behind it
    keys[g] = g < ng ? __float_as_uint((float)m) : 0u;
}

size_t tree_order_temp_bytes(int ng)
{
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, (const unsigned *)nullptr,
                                              (unsigned *)nullptr, (const int2 *)nullptr,
                                              (int2 *)nullptr, std::max(ng, 1));
    return bytes;
}

cudaError_t tree_order_groups(DevCount ng, const int2 *glist, int2 *ordered, const double *h2,
                              unsigned *keys_in, unsigned *keys_out, void *temp, size_t temp_bytes,
                              cudaStream_t st)
{
    if (ng.host <= 0) return cudaSuccess;
    k_tree_group_keys<<<(ng.host + 255) / 256, 256, 0, st>>>(ng, ng.host, glist, h2, keys_in);
    ++g_launches;
    size_t tb = temp_bytes;
    const cudaError_t e = cub::DeviceRadixSort::SortPairsDescending(temp, tb, keys_in, keys_out,
                                                                    glist, ordered, ng.host, 23,
                                                                    31, st);
    ++g_launches;
    return e != cudaSuccess ? e : cudaGetLastError();
}

size_t tree_acc_bytes(int nn) { return (size_t)nn * sizeof(NodeAcc); }

cudaError_t tree_props(DevCount nn, const TreeNode *nodes, const int *parent, int *done,
                       const SortedF64 &D, double theta, void *acc_buf, NodeGeom *geom, NodeMP *mp,
                       int sm_count, cudaStream_t st)
{
    k_tree_props<<<grid_for(nn, 8, sm_count * 16), 256, 0, st>>>(nn, nodes, parent, done, D, theta,
                                                            (NodeAcc *)acc_buf, geom, mp);
    ++g_launches;
    return cudaGetLastError();
}

int tree_walk_warps(int sm_count) { return sm_count * 8 * WALK_WARPS; }

cudaError_t tree_walk(const TreeWalkArgs &a, int sm_count, cudaStream_t st)
{
    if (a.nparts > 1)
        k_tree_walk<true><<<sm_count * 8, WALK_WARPS * 32, 0, st>>>(a);
    else
        k_tree_walk<false><<<sm_count * 8, WALK_WARPS * 32, 0, st>>>(a);
    ++g_launches;
    return cudaGetLastError();
}

int tree_scatter_blocks(int max_n)
{
    return std::max(1, std::min((max_n + SCATTER_NT - 1) / SCATTER_NT, 1024));
}

cudaError_t tree_scatter(const SetDesc *sets, int nsets, int max_n, int i_lo, int ni,
                         const double *res, const SortedF64 &D, const OutputsDev &out,
                         double *wpart, double *W, cudaStream_t st)
{
    const int nb = tree_scatter_blocks(max_n);
    k_tree_scatter<<<dim3(nb, grid_sets(nsets)), SCATTER_NT, 0, st>>>(
        sets, nsets, i_lo, ni, res, D, out, W ? wpart : nullptr);
    ++g_launches;
    if (W) {
        k_tree_wsum<<<nsets, SCATTER_NT, 0, st>>>(nb, wpart, W);
        ++g_launches;
    }
    return cudaGetLastError();
}

}  // namespace sg
