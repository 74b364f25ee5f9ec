// sg_noalloc.cu -- direct-summation FP64 forces for callers that cannot
// allocate device memory.
//
// Some callers cannot call cudaMalloc: code that runs while a CUDA graph is
// being captured, hosts that hand the GPU's memory to their own pool and
// forbid other allocations, or codes that must not add device allocations
// after start-up.  sphgrav_forces_fp64_noalloc serves them: the caller
// passes device inputs and outputs, and the only other memory the kernels
// use is the file-scope array below, which the CUDA runtime places in every
// GPU that loads this library and keeps there until the process exits.
//
// The kernel is the FP64 direct sum (same pair formulas and branch rule as
// the reference's CPU path, parallel_bleeding_edge/src/cpu_grav.f:46-157)
// on the caller's particle order, without the sorted layout the context API
// builds.  The j-range is split into chunks whose FP64 partial sums go to the
// static scratch; a second kernel adds them in chunk order, so the result is
// deterministic.
#include <algorithm>
#include <cmath>
#include "sg_launch.h"
#include "../../include/sphgrav_b200.h"

namespace sg {

constexpr int NA_NT = 128;   // threads per block
constexpr int NA_TJ = 128;   // sources staged per shared-memory tile
constexpr int NA_MIN_CHUNK = 256;  // sources of a chunk, at least
constexpr double NA_BIG = 1e150;   // |coordinate| up to which every r^2 is finite
constexpr size_t NA_SCRATCH_DOUBLES = SPHGRAV_NOALLOC_SCRATCH_BYTES / sizeof(double);

// High word that maybe_near compares r^2 with, for a particle at (x, y, z): its
// H^2's, or one above every r^2 (infinities and NaN too) past NA_BIG.
static __device__ __forceinline__ int na_limit(double x, double y, double z, double r2in)
{
    const bool fits = fabs(x) <= NA_BIG && fabs(y) <= NA_BIG && fabs(z) <= NA_BIG;
    return fits ? __double2hiint(fabs(r2in)) : 0x7fffffff;
}

// Partial sums [chunk][4][n].  Every element a call reads was written earlier
// in the same call, so nothing needs clearing between calls.
static __device__ __align__(256) double g_noalloc_scratch[NA_SCRATCH_DOUBLES];

// FP64 pair of rows i and sources j in the caller's order (no sorting):
// H^2 = |range2|, self-potential flag range2 > 0, lower index = min(i, j).
static __device__ __noinline__ PairOut pair_f64_raw(const double *x, const double *y,
                                                    const double *z, const double *m,
                                                    const double *r2in, int nkernel, int i, int j)
{
    const double dr1 = x[j] - x[i], dr2 = y[j] - y[i], dr3 = z[j] - z[i];
    const double r2 = SG_A(SG_A(SG_M(dr1, dr1), SG_M(dr2, dr2)), SG_M(dr3, dr3));
    const double amj = m[j];
    const double fourhpi2 = fabs(r2in[i]), fourhpj2 = fabs(r2in[j]);
    double gacc, gpot;
    if (r2 >= fmax(fourhpi2, fourhpj2)) {
        const double rinv = SG_D(1.0, __dsqrt_rn(r2));
        const double mrinv1 = SG_M(rinv, amj);
        gacc = SG_M(SG_M(rinv, rinv), mrinv1);
        gpot = -mrinv1;
    } else if (r2 > 0.0) {
        const double rinv = SG_D(1.0, __dsqrt_rn(r2));
        const double mrinv1 = SG_M(rinv, amj);
        const double twohpj = __dsqrt_rn(fourhpj2), mj12 = SG_D(amj, twohpj);
        near_kernel_f64(nkernel, r2, rinv, amj, __dsqrt_rn(fourhpi2), fourhpi2, twohpj, fourhpj2,
                        mj12, SG_D(mj12, fourhpj2), mrinv1, SG_M(SG_M(rinv, rinv), mrinv1), gacc,
                        gpot);
    } else {
        gacc = 0.0;
        const double twohpi = __dsqrt_rn(fourhpi2), twohpj = __dsqrt_rn(fourhpj2);
        const double s = SG_A(SG_D(amj, twohpi), SG_D(amj, twohpj));
        const double c = self_c(nkernel);
        if (i == j)
            gpot = r2in[i] > 0.0 ? SG_M(-c, s) : 0.0;
        else
            gpot = r2in[min(i, j)] > 0.0 ? SG_M(SG_M(-0.5, c), s) : 0.0;
    }
    PairOut o;
    o.ax = SG_M(gacc, dr1);
    o.ay = SG_M(gacc, dr2);
    o.az = SG_M(gacc, dr3);
    o.pot = gpot;
    return o;
}

// One block: NA_NT * K rows (K per thread) against one chunk of sources, staged
// in tiles of NA_TJ.  Pairs that may lie within max(H) leave the Newtonian sums
// (mass 0 at r = 1), are flagged 32 sources to a mask and join a queue per warp,
// which evaluates them 32 at a time, one pair per lane, with the CPU path's
// formulas; every owner then adds its own results in queue order
// (deterministic).  Pairs of a particle beyond NA_BIG join it too: r^2 may
// overflow, where rsqrt_f64 would give NaN.  The caller's order has no spatial meaning, so a warp meets
// a near pair every few sources: with the pairs evaluated where they are met,
// each cost the warp ~300 FP64-pipe instructions for one lane's sake.
template <int K>
__global__ void __launch_bounds__(NA_NT, K == 1 ? 4 : 3)
k_fp64_noalloc(int n, const double *x, const double *y, const double *z, const double *m,
               const double *r2in, int nkernel, int nchunks, double *part)
{
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NW = NA_NT / 32;
    __shared__ double s_x[NA_TJ], s_y[NA_TJ], s_z[NA_TJ], s_m[NA_TJ];
    __shared__ int s_h[NA_TJ];                    // na_limit of the sources
    __shared__ unsigned s_queue[NW][64];          // (source << 6) | row of the warp
    __shared__ unsigned s_owned[NW][K][32];       // entries of the round per owner
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int row0 = (blockIdx.x * NW + warp) * 32 * K;  // row (k, lane): row0 + 32 k + lane
    const int c = blockIdx.y;
    const int j0 = (int)((long long)n * c / nchunks), j1 = (int)((long long)n * (c + 1) / nchunks);
    bool act[K];
    double xi[K], yi[K], zi[K];
    int hih[K];
    double sum[K][4], acc[K][4];  // chunk sums; this tile's sums
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int i = row0 + 32 * k + lane;
        act[k] = i < n;
        xi[k] = act[k] ? x[i] : 1e15;
        yi[k] = act[k] ? y[i] : 1e15;
        zi[k] = act[k] ? z[i] : -1e15;
        hih[k] = act[k] ? na_limit(xi[k], yi[k], zi[k], r2in[i]) : 0;
        s_owned[warp][k][lane] = 0u;
#pragma unroll
        for (int q = 0; q < 4; q++) sum[k][q] = acc[k][q] = 0.0;
    }
    int pending = 0;  // queued pairs (uniform over the warp)
    __syncwarp();

    // evaluate the first cnt <= 32 queued pairs
    auto flush = [&](int cnt) {
        PairOut o{0.0, 0.0, 0.0, 0.0};
        if (lane < cnt) {
            const unsigned e = s_queue[warp][lane];
            const int r = e & 63u;
            o = pair_f64_raw(x, y, z, m, r2in, nkernel, row0 + r, (int)(e >> 6));
            atomicOr(&s_owned[warp][r >> 5][r & 31], 1u << lane);
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < K; k++) {
            unsigned own = s_owned[warp][k][lane];
            s_owned[warp][k][lane] = 0u;
            while (__any_sync(FULL, own != 0u)) {
                const int e = own ? __ffs(own) - 1 : 0;
                const double v[4] = {__shfl_sync(FULL, o.ax, e), __shfl_sync(FULL, o.ay, e),
                                     __shfl_sync(FULL, o.az, e), __shfl_sync(FULL, o.pot, e)};
                if (own) {
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[k][q] += v[q];
                }
                own &= own - 1u;
            }
        }
        __syncwarp();
        const unsigned v = 32 + lane < pending ? s_queue[warp][32 + lane] : 0u;
        __syncwarp();
        s_queue[warp][lane] = v;  // the rest (< 32 entries) moves to the front
        pending = max(0, pending - 32);
        __syncwarp();
    };

    double nx = 0.0, ny = 0.0, nz = 0.0, nm = 0.0, nh = 0.0;  // the next tile's source
    auto fetch = [&](int jt) {
        const int j = jt + tid;
        if (j < j1) {
            nx = x[j];
            ny = y[j];
            nz = z[j];
            nm = m[j];
            nh = r2in[j];
        }
    };
    static_assert(NA_NT == NA_TJ, "one staged source per thread");
    fetch(j0);
    for (int jt = j0; jt < j1; jt += NA_TJ) {
        __syncthreads();  // the previous tile has been read
        // sources past the chunk: mass 0 far from every row and from the idle rows
        const bool has = jt + tid < j1;
        s_x[tid] = has ? nx : 1e15;
        s_y[tid] = has ? ny : -1e15;
        s_z[tid] = has ? nz : 1e15;
        s_m[tid] = has ? nm : 0.0;
        s_h[tid] = has ? na_limit(nx, ny, nz, nh) : 0;
        __syncthreads();
        fetch(jt + NA_TJ);
        const int blocks = min(NA_TJ / 32, (j1 - jt + 31) / 32);
        for (int b = 0; b < blocks; b++) {
            unsigned mk[K];
#pragma unroll
            for (int k = 0; k < K; k++) mk[k] = 0u;
#pragma unroll 4  // 20,011 particles: 691 us against 719 with 2
            for (int u = 0; u < 32; u++) {
                const int j = 32 * b + u;
                const double xj = s_x[j], yj = s_y[j], zj = s_z[j], mj = s_m[j];
                const int hj = s_h[j];
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const double dx = xj - xi[k], dy = yj - yi[k], dz = zj - zi[k];
                    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
                    const bool nr = maybe_near(r2, max(hih[k], hj));
                    if (nr) mk[k] |= 1u << u;
                    const double rinv = rsqrt_f64(nr ? 1.0 : r2);
                    const double mr = (nr ? 0.0 : mj) * rinv;
                    const double mr3 = mr * (rinv * rinv);
                    acc[k][0] = fma(mr3, dx, acc[k][0]);
                    acc[k][1] = fma(mr3, dy, acc[k][1]);
                    acc[k][2] = fma(mr3, dz, acc[k][2]);
                    acc[k][3] -= mr;
                }
            }
            const int left = j1 - (jt + 32 * b);  // a padding source is never queued
            const unsigned valid = left >= 32 ? FULL : (1u << left) - 1u;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const unsigned mine = act[k] ? mk[k] & valid : 0u;
                unsigned any = __reduce_or_sync(FULL, mine);
                while (any) {
                    const int u = __ffs(any) - 1;
                    any &= any - 1u;
                    const unsigned who = __ballot_sync(FULL, (mine >> u) & 1u);
                    if ((mine >> u) & 1u)
                        s_queue[warp][pending + __popc(who & below)] =
                            ((unsigned)(jt + 32 * b + u) << 6) | (unsigned)(32 * k + lane);
                    pending += __popc(who);
                    __syncwarp();
                    if (pending >= 32) flush(32);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                sum[k][q] += acc[k][q];
                acc[k][q] = 0.0;
            }
        }
    }
    if (pending > 0) flush(pending);
#pragma unroll
    for (int k = 0; k < K; k++) {
        if (!act[k]) continue;
        double *p = part + (size_t)c * 4 * n + row0 + 32 * k + lane;
#pragma unroll
        for (int q = 0; q < 4; q++) p[(size_t)q * n] = sum[k][q] + acc[k][q];
    }
}

__global__ void k_merge_noalloc(int n, int nchunks, const double *part, double *ax, double *ay,
                                double *az, double *pot)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int c = 0; c < nchunks; c++)
        for (int q = 0; q < 4; q++) s[q] += part[((size_t)c * 4 + q) * n + i];
    ax[i] = s[0];
    ay[i] = s[1];
    az[i] = s[2];
    pot[i] = s[3];
}

}  // namespace sg

using namespace sg;

// Device address of the static scratch, looked up once per device.  Atomic:
// host threads calling on different devices (or racing on the first call of
// one device, which both resolve to the same address) must not race.
static std::atomic<void *> g_noalloc_ptr[64];

// Blocks of the K = k kernel resident on the device, looked up once per device.
static int noalloc_resident(int dev, int k)
{
    static std::atomic<int> cache[64][2];
    int v = cache[dev][k - 1].load(std::memory_order_acquire);
    if (v == 0) {
        int sms = 0, per = 0;
        const void *f = k == 2 ? (const void *)k_fp64_noalloc<2> : (const void *)k_fp64_noalloc<1>;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, NA_NT, 0) != cudaSuccess) {
            cudaGetLastError();
            return 148;
        }
        v = std::max(1, sms * per);
        cache[dev][k - 1].store(v, std::memory_order_release);
    }
    return v;
}

extern "C" int sphgrav_forces_fp64_noalloc(int n, const double *x, const double *y,
                                           const double *z, const double *mass,
                                           const double *range2, int nkernel, double *ax,
                                           double *ay, double *az, double *pot, void *stream)
{
    if (n < 0 || nkernel < 0 || nkernel > 2) return SPHGRAV_ERR_INVALID_ARGUMENT;
    if (n > SPHGRAV_NOALLOC_MAX_N) return SPHGRAV_ERR_TOO_LARGE;
    if (n == 0) return SPHGRAV_OK;
    if (!x || !y || !z || !mass || !range2 || !ax || !ay || !az || !pot)
        return SPHGRAV_ERR_INVALID_ARGUMENT;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return SPHGRAV_ERR_NO_DEVICE;
    }
    void *part_p = g_noalloc_ptr[dev].load(std::memory_order_acquire);
    if (!part_p) {
        // set-up on this device's first call: the scratch's device address (host
        // code cannot use the symbol's name as one), and everything that a call of
        // another size would otherwise load or ask for inside a capture
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        for (const void *f : {(const void *)k_fp64_noalloc<1>, (const void *)k_fp64_noalloc<2>,
                              (const void *)k_merge_noalloc}) {
            cudaFuncAttributes at;
            if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, f);
        }
        for (int k = 1; k <= 2; k++) noalloc_resident(dev, k);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return SPHGRAV_ERR_CUDA;
        }
        g_noalloc_ptr[dev].store(p, std::memory_order_release);
        part_p = p;
    }
    double *part = (double *)part_p;
    // Rows per thread and source chunks: two rows per thread from 16,384
    // particles (the source loads then serve two rows), and the chunk count,
    // within the scratch and at least NA_MIN_CHUNK sources each, whose blocks
    // fill the last wave best (ties: fewer chunks).
    const int k = n >= 16384 ? 2 : 1;
    const int rows = NA_NT * k;
    const long long row_blocks = (n + rows - 1) / rows;
    const int resident = noalloc_resident(dev, k);
    const int most = (int)std::max<long long>(
        1, std::min<long long>({64, (long long)NA_SCRATCH_DOUBLES / (4ll * n), n / NA_MIN_CHUNK}));
    int nchunks = 1;
    double best = -1.0;
    for (int c = 1; c <= most; c++) {
        const double waves = (double)row_blocks * c / resident;
        const double eff = waves / std::ceil(waves) - 0.002 * c;
        if (eff > best + 1e-9) {
            best = eff;
            nchunks = c;
        }
    }
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid((unsigned)row_blocks, nchunks);
    if (k == 2)
        k_fp64_noalloc<2><<<grid, NA_NT, 0, st>>>(n, x, y, z, mass, range2, nkernel, nchunks, part);
    else
        k_fp64_noalloc<1><<<grid, NA_NT, 0, st>>>(n, x, y, z, mass, range2, nkernel, nchunks, part);
    k_merge_noalloc<<<(n + 255) / 256, 256, 0, st>>>(n, nchunks, part, ax, ay, az, pot);
    g_launches += 2;
    if (cudaGetLastError() != cudaSuccess) return SPHGRAV_ERR_CUDA;
    return SPHGRAV_OK;
}
