// diag.cu — FP64 conserved-quantity diagnostics of a body set.
//
// The reference has none; the engine states its energy drift against these:
//   M = sum m, centre of mass and its velocity, P = sum m v,
//   L = sum m (x cross v) about the origin, T = sum m v^2 / 2,
//   W = -(G/2) sum_{i != j} m_i m_j / sqrt(|x_i - x_j|^2 + eps^2)
// (the Plummer-softened potential whose gradient is the walk's force law).
// Every sum is in double precision; W is the exact O(N^2) pair sum.  Block
// partials are reduced by one block in a fixed order, so results are
// deterministic for a given launch geometry.
#include <type_traits>

#include "bh_internal.cuh"
#include "rsqrt64.cuh"

namespace {
constexpr int kThreads = 256;
constexpr int kMoments = 11;  // M, Mx, My, Mz, Px, Py, Pz, Lx, Ly, Lz, 2T
constexpr int kMomentBlocksMax = 1184;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block sum of v[0..K); result in thread 0.
template <int K, int Threads = kThreads>
__device__ void block_sum(double v[K]) {
    __shared__ double part[Threads / 32][K];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = warp_sum(v[k]);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; k++) part[w][k] = v[k];
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = warp_sum(lane < Threads / 32 ? part[lane][k] : 0.0);
    }
    __syncthreads();
}
}  // namespace

__global__ void __launch_bounds__(kThreads)
k_diag_moments(const float4* __restrict__ pos, const float3* __restrict__ vel, int n, double* __restrict__ partial) {
    double v[kMoments] = {0};
    for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        const float4 p = pos[i];
        const float3 u = vel[i];
        const double m = p.w, x = p.x, y = p.y, z = p.z, vx = u.x, vy = u.y, vz = u.z;
        v[0] += m;
        v[1] += m * x;
        v[2] += m * y;
        v[3] += m * z;
        v[4] += m * vx;
        v[5] += m * vy;
        v[6] += m * vz;
        v[7] += m * (y * vz - z * vy);
        v[8] += m * (z * vx - x * vz);
        v[9] += m * (x * vy - y * vx);
        v[10] += m * (vx * vx + vy * vy + vz * vz);
    }
    block_sum<kMoments>(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < kMoments; k++) partial[(size_t)blockIdx.x * kMoments + k] = v[k];
}

// The pair sum, every unordered pair once.  Bodies in rows of 256 (two per
// thread); row r meets itself (pairs i < j) and the next rows/2 rows round the
// circle (when the number of rows is even, the row opposite only from its first
// half), so that all rows do the same work; block (r, y) takes part y of the
// row's tiles and writes sum m_i sum_j m_j / r_ij (softened).  FP64 pipe bound
// as the direct sum is, 13 operations a pair: 65,537 bodies 7.6 -> 2.2 ms, 1M 1180 -> 436,
// against one ordered pair at a time, one target per thread.  A block whose sum is
// not finite takes it again with rsqrt() (1M with a body at infinity: 588, 1176 before).
constexpr int kPotThreads = 128;
constexpr int kRow = 2 * kPotThreads;

__global__ void __launch_bounds__(kPotThreads, 8)
k_diag_potential(const float4* __restrict__ pos, int n, int rows, int perPart, double eps2, double* __restrict__ partial) {
    __shared__ double2 tile[kRow][2];  // (x, y), (z, m)
    const int row = blockIdx.x;
    int id[2];
    double x[2], y[2], z[2], m[2], phi[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        id[k] = row * kRow + k * kPotThreads + threadIdx.x;
        const float4 p = id[k] < n ? pos[id[k]] : make_float4(0.f, 0.f, 0.f, 0.f);
        x[k] = p.x; y[k] = p.y; z[k] = p.z; m[k] = p.w;
    }
    const int most = rows / 2;  // tiles at distance 0 .. most
    const int lo = blockIdx.y * perPart, hi = lo + perPart < most + 1 ? lo + perPart : most + 1;
    auto sum = [&](auto edges) {
        phi[0] = phi[1] = 0.0;
        for (int d = lo; d < hi; d++) {
            if (d > 0 && 2 * d == rows && row >= d) break;  // the opposite row has this pair
            const int other = row + d < rows ? row + d : row + d - rows;
            const int base = other * kRow, cnt = n - base < kRow ? n - base : kRow;
            __syncthreads();
            for (int j = threadIdx.x; j < cnt; j += kPotThreads) {
                const float4 p = pos[base + j];
                tile[j][0] = make_double2(p.x, p.y);
                tile[j][1] = make_double2(p.z, p.w);
            }
            __syncthreads();
            auto add = [&](int j, bool own) {
                const double2 xy = tile[j][0], zm = tile[j][1];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const double dx = xy.x - x[k], dy = xy.y - y[k], dz = zm.x - z[k];
                    const double r2 = fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2)));
                    double t;
                    if (decltype(edges)::value) {  // half of either body's share: they differ where a mass is 0 or infinite
                        const double ri = rsqrt(r2);
                        t = 0.5 * (m[k] * (zm.y * ri) + zm.y * (m[k] * ri));
                    } else {
                        t = mass_over_r(zm.y, r2);
                    }
                    phi[k] += own && base + j <= id[k] ? 0.0 : t;
                }
            };
            if (d == 0) {
                for (int j = 0; j < cnt; j++) add(j, true);
            } else if (decltype(edges)::value) {
#pragma unroll 1
                for (int j = 0; j < cnt; j++) add(j, false);
            } else {
#pragma unroll 4
                for (int j = 0; j < cnt; j++) add(j, false);
            }
        }
        const double f0 = decltype(edges)::value ? phi[0] : m[0] * phi[0], f1 = decltype(edges)::value ? phi[1] : m[1] * phi[1];
        return (id[0] < n ? f0 : 0.0) + (id[1] < n ? f1 : 0.0);
    };
    double v[1] = {sum(std::false_type())};
    // a pair at distance 0 or infinity, a mass that is not finite, a softening
    // whose square is subnormal: once more with rsqrt()
    if (__syncthreads_or(!isfinite(v[0])) && n > 1) v[0] = sum(std::true_type());
    block_sum<1, kPotThreads>(v);
    if (threadIdx.x == 0) partial[(size_t)blockIdx.y * rows + row] = v[0];
}

// One block: fixed-order reduction of the partials into the result
// (kMoments moment sums, then the sum over unordered pairs).
__global__ void __launch_bounds__(kThreads)
k_diag_finalize(const double* __restrict__ moments, int nMomentBlocks, const double* __restrict__ pot, int nPotBlocks,
                double* __restrict__ out) {
    double v[kMoments + 1] = {0};
    for (int b = threadIdx.x; b < nMomentBlocks; b += kThreads)
        for (int k = 0; k < kMoments; k++) v[k] += moments[(size_t)b * kMoments + k];
    for (int b = threadIdx.x; b < nPotBlocks; b += kThreads) v[kMoments] += pot[b];
    block_sum<kMoments + 1>(v);
    if (threadIdx.x == 0)
        for (int k = 0; k <= kMoments; k++) out[k] = v[k];
}

extern "C" int bh_diagnostics_f64(const float4* pos, const float3* vel, int n, double eps, double G, int withPotential,
                                  bh_diagnostics* out, cudaStream_t s) {
    if (!pos || !vel || !out || n <= 0) return BH_ERR_INVALID;
    int mBlocks = (n + kThreads - 1) / kThreads;
    mBlocks = mBlocks > kMomentBlocksMax ? kMomentBlocksMax : mBlocks;
    // rows of the pair sum, each split so that about four waves of eight blocks
    // per SM are there in all
    const int rows = (n - 1) / kRow + 1;
    int parts = (32 * bh_sm_count() + rows - 1) / rows;
    parts = parts > rows / 2 + 1 ? rows / 2 + 1 : parts;
    const int perPart = (rows / 2 + parts) / parts;
    parts = rows / 2 / perPart + 1;
    const int pBlocks = withPotential ? rows * parts : 0;
    double* scratch = nullptr;
    const size_t words = (size_t)mBlocks * kMoments + pBlocks + kMoments + 1;
    cudaError_t e = cudaMallocAsync(&scratch, words * sizeof(double), s);
    if (e != cudaSuccess) return bh_note_cuda_error(e);
    double* mPart = scratch;
    double* pPart = mPart + (size_t)mBlocks * kMoments;
    double* res = pPart + pBlocks;
    double h[kMoments + 1];
    k_diag_moments<<<mBlocks, kThreads, 0, s>>>(pos, vel, n, mPart);
    if (withPotential)
        k_diag_potential<<<dim3(rows, parts), kPotThreads, 0, s>>>(pos, n, rows, perPart, eps * eps, pPart);
    k_diag_finalize<<<1, kThreads, 0, s>>>(mPart, mBlocks, pPart, pBlocks, res);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, res, sizeof h, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaFreeAsync(scratch, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bh_note_cuda_error(e);
    bh_diagnostics d;
    d.mass = h[0];
    const double inv = h[0] != 0.0 ? 1.0 / h[0] : 0.0;
    for (int k = 0; k < 3; k++) {
        d.com[k] = h[1 + k] * inv;
        d.momentum[k] = h[4 + k];
        d.comVel[k] = h[4 + k] * inv;
        d.angularMomentum[k] = h[7 + k];
    }
    d.kinetic = 0.5 * h[10];
    d.potential = withPotential ? -G * h[11] : 0.0;
    d.total = d.kinetic + d.potential;
    *out = d;
    return BH_OK;
}
