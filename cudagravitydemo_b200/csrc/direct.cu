// direct.cu — FP64 direct-sum accelerations of selected target bodies.
//
// The error of every Barnes-Hut walk is stated against this sum:
// a_t = sum_j G m_j (x_j - x_t) / (|x_j - x_t|^2 + eps^2)^{3/2} in double
// precision over all n source bodies.  It is an evaluation tool (labels for the
// learned opening criterion, RMS force errors), not part of a step.
//
// What bounds it: the FP64 pipe, 16 operations a pair (one warp instruction
// every 2 cycles and sub-partition): 29.5 ms for 3.4e10 pairs.  Sources are
// converted to double once per tile instead of once per pair, each lane has two
// targets (one load of a source serves both), and the sources of a target are
// split over the block's warps and over a cluster of up to 8 blocks, whose
// partial sums meet in shared memory in a fixed order, so that a few hundred
// targets keep the GPU busy too and no scratch memory is needed.  1M sources:
// 32,768 targets 105.7 -> 35.6 ms, 2,048 targets 105.7 -> 2.7 ms.
// A block whose sums are not finite takes them again term by term (63.7 ms with a
// body at infinity, 106.0 by the sum before).
#include <cooperative_groups.h>

#include "bh_internal.cuh"
#include "rsqrt64.cuh"

namespace cg = cooperative_groups;

namespace {
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTargets = 64;       // per block, two per lane
constexpr int kTile = 2 * kThreads;  // sources in shared memory, kTile / kWarps per warp
constexpr int kMaxSplit = 8;       // blocks of a cluster (the portable most)

// Sources [base, base + kTile) into the tile; how many there are.
__device__ __forceinline__ int load_tile(const float4* __restrict__ pos, int n, long long base, double2 (*tile)[2]) {
    const int cnt = n - base < kTile ? (int)(n - base) : kTile;
    __syncthreads();
    for (int j = threadIdx.x; j < cnt; j += kThreads) {
        const float4 p = pos[base + j];
        tile[j][0] = make_double2(p.x, p.y);
        tile[j][1] = make_double2(p.z, p.w);
    }
    __syncthreads();
    return cnt;
}

// A warp's share of the sum at (x, y, z) term by term, whatever the terms are.
__device__ __forceinline__ double3 plain_sum(const float4* pos, int n, int rank, int size, double2 (*tile)[2], double x,
                                             double y, double z, double eps2) {
    double3 a = make_double3(0.0, 0.0, 0.0);
    for (long long base = (long long)rank * kTile; base < n; base += (long long)size * kTile) {
        const int cnt = load_tile(pos, n, base, tile);
        for (int j = threadIdx.x >> 5; j < cnt; j += kWarps) {
            const double2 xy = tile[j][0], zm = tile[j][1];
            const double dx = xy.x - x, dy = xy.y - y, dz = zm.x - z;
            const double ri = rsqrt(fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2))));
            const double f = zm.y * ri * ri * ri;
            a.x = fma(f, dx, a.x);
            a.y = fma(f, dy, a.y);
            a.z = fma(f, dz, a.z);
        }
    }
    return a;
}
}  // namespace

// Cluster c = targets [64 c, +64); its block r takes the source tiles r, r + size, ...
// eps2: the softening's square; soft2: the same for the series, which wants it
// finite (an argument of its own: formed in the kernel it cost 1%, 36.0 ms).
__global__ void __launch_bounds__(kThreads, 4)
k_direct_f64(const float4* __restrict__ pos, int n, const int* __restrict__ targets, int nt, double eps2, double soft2,
             double G, double* __restrict__ acc) {
    __shared__ double2 tile[kTile][2];  // (x, y), (z, m)
    __shared__ double part[kWarps][3][kTargets];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), size = (int)cluster.num_blocks();
    const int t0 = (int)(blockIdx.x / size) * kTargets;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double x[2], y[2], z[2], ax[2], ay[2], az[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int t = t0 + lane + 32 * k;
        const float4 p = t < nt ? pos[targets ? targets[t] : t] : make_float4(0.f, 0.f, 0.f, 0.f);
        x[k] = p.x; y[k] = p.y; z[k] = p.z;
        ax[k] = ay[k] = az[k] = 0.0;
    }
    for (long long base = (long long)rank * kTile; base < n; base += (long long)size * kTile) {
        const int cnt = load_tile(pos, n, base, tile);
#pragma unroll 4
        for (int j = w; j < cnt; j += kWarps) {
            const double2 xy = tile[j][0], zm = tile[j][1];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const double dx = xy.x - x[k], dy = xy.y - y[k], dz = zm.x - z[k];
                const double r2 = fma(dz, dz, fma(dy, dy, fma(dx, dx, soft2)));
                const double f = mass_over_r3(zm.y, r2);
                ax[k] = fma(f, dx, ax[k]);
                ay[k] = fma(f, dy, ay[k]);
                az[k] = fma(f, dz, az[k]);
            }
        }
    }
    // not finite: a body or mass that is not, or a softening whose square is
    // subnormal; once more with rsqrt().  (Without softening a target, a source
    // itself, comes out as NaN either way.)
    bool fine = true;
#pragma unroll
    for (int k = 0; k < 2; k++) fine = fine && isfinite(ax[k]) && isfinite(ay[k]) && isfinite(az[k]);
    if (__syncthreads_or(!fine) && eps2 != 0.0)
        for (int k = 0; k < 2; k++) {
            const double3 r = plain_sum(pos, n, rank, size, tile, x[k], y[k], z[k], eps2);
            ax[k] = r.x; ay[k] = r.y; az[k] = r.z;
        }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        part[w][0][lane + 32 * k] = ax[k];
        part[w][1][lane + 32 * k] = ay[k];
        part[w][2][lane + 32 * k] = az[k];
    }
    __syncthreads();
    // the warps' sums in part[0], then the blocks' in rank order
    double* const mine = &part[0][0][0];
    if (threadIdx.x < 3 * kTargets) {
        double s = mine[threadIdx.x];
        for (int k = 1; k < kWarps; k++) s += mine[k * 3 * kTargets + threadIdx.x];
        mine[threadIdx.x] = s;
    }
    cluster.sync();
    if (rank == 0 && threadIdx.x < 3 * kTargets) {
        double s = mine[threadIdx.x];
        for (int k = 1; k < size; k++) s += cluster.map_shared_rank(mine, k)[threadIdx.x];
        const int axis = threadIdx.x / kTargets, t = t0 + threadIdx.x % kTargets;
        if (t < nt) acc[3 * (size_t)t + axis] = G * s;
    }
    cluster.sync();  // no block leaves while its sums are read
}

extern "C" int bh_direct_sum_f64(const float4* pos, int n, const int* targets, int ntargets, double eps, double G,
                                 double* acc, cudaStream_t s) {
    if (!pos || !acc || n <= 0 || ntargets <= 0) return BH_ERR_INVALID;
    const int groups = (ntargets + kTargets - 1) / kTargets;
    // blocks per target group: the fewest of 1, 2, 4, 8 that give eight waves
    // of the four blocks an SM holds (the last wave is then an eighth at most),
    // and no more than there are tiles
    int split = 1;
    while (split < kMaxSplit && (long long)groups * split < 32ll * bh_sm_count() && (long long)split * kTile < n)
        split *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)groups * (unsigned)split);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)split;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // (from 1e300 on every term of a finite mass is 0 in double precision)
    const double eps2 = eps * eps, soft2 = eps2 < 1e300 || eps2 != eps2 ? eps2 : 1e300;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_direct_f64, pos, n, targets, ntargets, eps2, soft2, G, acc);
    return e == cudaSuccess ? BH_OK : bh_note_cuda_error(e);
}
