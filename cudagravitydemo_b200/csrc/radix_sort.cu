// radix_sort.cu — stable LSD radix sort of (uint64 key, uint32 value) pairs
// for sm_100a.
//
// Replaces the reference's CUB DeviceRadixSort::SortPairs call
// (sorting.cu:15-92).  Same contract: stable, ascending, inputs untouched,
// results in separate buffers.  Design: "onesweep" (Adinets & Merrill 2022):
//   - one histogram read of the keys gives every digit's global counts
//     (fused into the Morton kernel when the sort follows it);
//   - one kernel per 8-bit digit: each CTA takes the next tile from an atomic
//     counter, ranks its keys stably warp by warp, publishes its
//     per-digit counts, and computes the count of each digit in all earlier
//     tiles by decoupled look-back; it then scatters through shared memory so
//     that each digit's run is written contiguously;
//   - each pass after the first is a programmatic dependent launch of the one
//     before: its tiles are scheduled while the previous pass drains and wait
//     for it only before loading their keys.
// Look-back waits are bounded (BH_SPIN_LIMIT polls): a wait that gives up sets
// BH_ERR_TIMEOUT in the error word instead of hanging.
#include <cooperative_groups.h>

#include "bh_internal.cuh"
#include "bh_kernels.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;                 // keys per thread
constexpr int kTile = kThreads * kItems;  // 4096 keys per tile
constexpr uint32_t kFlagAgg = 1u << 30;     // tile count published
constexpr uint32_t kFlagPrefix = 2u << 30;  // inclusive prefix published
constexpr uint32_t kValueMask = (1u << 30) - 1u;
#ifndef BH_SORT_LOOKBACK
#define BH_SORT_LOOKBACK 8
#endif
constexpr int kLookback = BH_SORT_LOOKBACK;  // predecessor tiles read per look-back round trip

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_volatile(uint32_t* p, uint32_t v) {
    asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Decoupled look-back for one digit: the count of that digit in tiles
// 0..tile-1, read from status (one word per tile and digit, stride 256).  A
// window of kLookback predecessors is loaded per round trip (independent
// loads), then consumed in tile order until a published prefix (done) or an
// unpublished tile (wait on it).  The wait is bounded: after BH_SPIN_LIMIT
// round trips without progress it sets BH_ERR_TIMEOUT and returns what it
// has, so a tile that never publishes cannot hang the sort.
__device__ __forceinline__ uint32_t lookback_exclusive(const uint32_t* status, int tile, int d, int* err) {
    uint32_t excl = 0;
    int j = tile - 1;
    unsigned spins = 0;
    while (j >= 0) {
        uint32_t v[kLookback];
#pragma unroll
        for (int k = 0; k < kLookback; k++)
            v[k] = (j - k >= 0) ? ld_volatile(status + (size_t)(j - k) * 256 + d) : kFlagPrefix;
        bool done = false;
        int k = 0;
#pragma unroll
        for (; k < kLookback; k++) {
            const uint32_t flag = v[k] & ~kValueMask;
            if (flag == 0u) break;
            excl += v[k] & kValueMask;
            if (flag == kFlagPrefix) {
                done = true;
                break;
            }
        }
        if (done) break;
        j -= k;  // k < kLookback: tile j - k has published nothing yet
        if (k < kLookback && ++spins > BH_SPIN_LIMIT) {
            bh_set_error(err, BH_ERR_TIMEOUT);
            break;
        }
    }
    return excl;
}

}  // namespace

// Upfront digit histogram for a standalone sort: counts digits 0..npass-1 of
// every key into hist[npass][256] (must be zero on entry).  Eight copies of
// each bin in neighbouring banks (lane mod 8 takes its own), so that a warp
// whose keys share a digit, as sorted or clustered keys do, waits four times
// and not 32 times for one bin: 298 -> 60 us at 16.8M clustered
// keys.
constexpr int kHistCopies = 8;
constexpr int kHistThreads = 512;
__global__ void __launch_bounds__(kHistThreads)
k_sort_histogram(const uint64_t* __restrict__ keys, int n, uint32_t* __restrict__ hist, int npass) {
    extern __shared__ uint32_t sh[];  // [npass][256][kHistCopies]
    const int bins = npass * 256;
    for (int i = threadIdx.x; i < bins * kHistCopies; i += kHistThreads) sh[i] = 0u;
    __syncthreads();
    const int stride = gridDim.x * kHistThreads;
    uint32_t* mine = sh + (threadIdx.x & (kHistCopies - 1));
    auto count = [&](uint64_t k) {
        for (int p = 0; p < npass; p++) {
            atomicAdd(mine + (p * 256 + (int)(k & 255u)) * kHistCopies, 1u);
            k >>= 8;
        }
    };
    int i = blockIdx.x * kHistThreads + threadIdx.x;
    for (; i + 3 * (long long)stride < n; i += 4 * stride) {  // four loads in flight
        const uint64_t a = __ldg(&keys[i]), b = __ldg(&keys[i + stride]);
        const uint64_t c = __ldg(&keys[i + 2 * stride]), d = __ldg(&keys[i + 3 * stride]);
        count(a);
        count(b);
        count(c);
        count(d);
    }
    for (; i < n; i += stride) count(__ldg(&keys[i]));
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += kHistThreads) {
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < kHistCopies; k++) c += sh[b * kHistCopies + k];
        if (c) atomicAdd(&hist[b], c);
    }
}

// One digit pass.  hist: the 256 global counts of this digit.  status:
// [numTiles][256] words, zero on entry.  tileCounter: zero on entry.
// identityVals: the values are the input positions (valsIn is not read).
//
// A pass is bound by the chain of phases of one tile (loads, ranks, offsets,
// look-back, scatter, stores) and then by shared-memory wavefronts (57% of
// peak), not by HBM (0.45 of the copy rate at 16.8M), so a tile has many
// threads with few keys each: 512 x 8 keys, two tiles per SM.  Ranks by a mask
// per digit in shared memory instead of 8 ballots halve the instructions (194
// -> 124 per 32 keys).  The second half of the threads looks back over the
// earlier tiles while the first half already scatters, and the values are only
// loaded for the scatter (registers).  Standalone sort of 63-bit keys at 16.8M
// pairs 1638 -> 1152 us, 4.2M 464 -> 324, 1M 160 -> 110, 16,384 80 -> 57; the
// step's sort stage at 1M 135 -> 105.  Measured and not kept: 3 tiles per SM
// (40 registers, spills: 1234 us at 16.8M, 136 at 1M), 12 keys per thread
// (1097 and 127), values loaded before the look-back (1160 and 111).
__global__ void __launch_bounds__(kThreads, 2)
k_sort_pass(const uint64_t* __restrict__ keysIn, const uint32_t* __restrict__ valsIn,
            uint64_t* __restrict__ keysOut, uint32_t* __restrict__ valsOut, int n, int shift,
            const uint32_t* __restrict__ hist, uint32_t* status, int* tileCounter, int* err,
            int identityVals) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* skeys = reinterpret_cast<uint64_t*>(smem);           // kTile
    uint32_t* svals = reinterpret_cast<uint32_t*>(skeys + kTile);  // kTile
    uint32_t* warpHist = svals + kTile;                            // [kWarps][256]
    uint32_t* warpMask = reinterpret_cast<uint32_t*>(smem);        // [kWarps][256]: lanes of a digit (before skeys is filled)
    uint32_t* localStart = warpHist + kWarps * 256;                // [256]
    uint32_t* tileCounts = localStart + 256;                       // [256]
    uint32_t* target = tileCounts + 256;                           // [256]: output position of tile position 0
    __shared__ int sTile;
    __shared__ uint32_t baseSum[8], countSum[8];

    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    // programmatic dependent launch: the next pass may be scheduled once every
    // tile of this one runs, and its prologue (tile id, digit bases from the
    // upfront histograms) overlaps this pass's tail
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) sTile = atomicAdd(tileCounter, 1);
    for (int i = tid; i < kWarps * 256; i += kThreads) {
        warpHist[i] = 0u;
        warpMask[i] = 0u;
    }
    // exclusive scan over one digit per thread (the first 256 threads), in
    // two steps around a barrier
    auto scanWarp = [&](uint32_t c, uint32_t* sums) {
        uint32_t x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) sums[w] = x;
        return x - c;
    };
    auto scanBlock = [&](uint32_t x, const uint32_t* sums) {
        for (int k = 0; k < w; k++) x += sums[k];
        return x;
    };
    uint32_t digitBase = 0;  // first output position of digit tid
    if (tid < 256) digitBase = scanWarp(hist[tid], baseSum);
    __syncthreads();
    if (tid < 256) target[tid] = scanBlock(digitBase, baseSum);  // (read back by the thread that looks back)
    const int tile = sTile;
    const int tileBase = tile * kTile;
    const int tileValid = n - tileBase < kTile ? n - tileBase : kTile;
    // the keys are the previous pass's output: wait for that grid to complete
    // (returns at once for a launch without a programmatic dependency)
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // load: warp w owns keys [tileBase + w*32*kItems, +32*kItems), item k of
    // lane l at offset k*32 + l (coalesced, and in input order k-major).  Past
    // the end come keys of the highest digit: last in order, so they rank
    // behind every key of the last tile and are never written out
    uint64_t key[kItems];
    uint32_t rank[kItems];
    const int warpOff = w * 32 * kItems + lane;
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const int i = warpOff + k * 32;
        key[k] = i < tileValid ? keysIn[tileBase + i] : ~0ull;
    }
    auto digit = [&](int k) { return (uint32_t)(key[k] >> shift) & 255u; };
    // stable ranks within the warp, items in order.  The lanes with the same
    // digit meet in a mask per digit in shared memory (one atomic OR each);
    // a warp whose keys all share the digit, as nearly sorted keys do in the
    // high digits, is spared the 32 turns at one word
    uint32_t* myHist = warpHist + w * 256;
    uint32_t* myMask = warpMask + w * 256;
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const uint32_t d = digit(k);
        uint32_t peers = 0xffffffffu, before;
        if (__all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {
            before = myHist[d];
            __syncwarp();
            if (lane == 0) myHist[d] = before + 32u;
        } else {
            atomicOr(&myMask[d], 1u << lane);
            __syncwarp();
            peers = myMask[d];
            before = myHist[d];
            __syncwarp();
            if ((peers & lt) == 0u) {  // the lowest peer moves the counter and clears the mask
                myHist[d] = before + __popc(peers);
                myMask[d] = 0u;
            }
        }
        rank[k] = before + __popc(peers & lt);
        __syncwarp();
    }
    __syncthreads();
    // per digit: tile total, published at once; then where each warp's keys of
    // the digit start in the tile
    uint32_t c[kWarps], start = 0, total = 0;
    if (tid < 256) {
#pragma unroll
        for (int k = 0; k < kWarps; k++) c[k] = warpHist[k * 256 + tid];
#pragma unroll
        for (int k = 0; k < kWarps; k++) total += c[k];
        st_volatile(status + (size_t)tile * 256 + tid, (tile == 0 ? kFlagPrefix : kFlagAgg) | total);
        start = scanWarp(total, countSum);
    }
    __syncthreads();
    if (tid < 256) {
        start = scanBlock(start, countSum);
        localStart[tid] = start;
        tileCounts[tid] = total;
#pragma unroll
        for (int k = 0; k < kWarps; k++) {
            warpHist[k * 256 + tid] = start;
            start += c[k];
        }
    }
    __syncthreads();
    if (tid >= 256) {  // look back over earlier tiles
        const int d = tid - 256;
        uint32_t excl = 0;
        if (tile > 0) {
            excl = lookback_exclusive(status, tile, d, err);
            st_volatile(status + (size_t)tile * 256 + d, kFlagPrefix | ((excl + tileCounts[d]) & kValueMask));
        }
        target[d] += excl - localStart[d];
    }
    // scatter into shared memory in sorted-within-tile order
    uint32_t val[kItems];
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const int i = warpOff + k * 32;
        val[k] = 0u;
        if (i < tileValid) val[k] = identityVals ? (uint32_t)(tileBase + i) : valsIn[tileBase + i];
    }
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const uint32_t p = myHist[digit(k)] + rank[k];
        skeys[p] = key[k];
        svals[p] = val[k];
    }
    __syncthreads();
    // write out: consecutive positions of a digit go to consecutive addresses
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const int j = tid + k * kThreads;
        if (j < tileValid) {
            const uint64_t q = skeys[j];
            const uint32_t dst = target[(uint32_t)(q >> shift) & 255u] + (uint32_t)j;
            keysOut[dst] = q;
            valsOut[dst] = svals[j];
        }
    }
}

// Every pass of a small sort in one launch of one cluster.  The keys stay in
// the blocks' shared memory: block b holds positions [b * 1024 Items, + 1024
// Items).  A pass ranks each block's keys as k_sort_pass does, the blocks read
// each other's digit counts, and every key is stored into the block that holds
// its new position (distributed shared memory); the last pass stores to global
// memory.  No histogram, no look-back, no status words; a pass costs two
// cluster barriers (about 1 us each, what bounds it) instead of a launch and a
// chain of tiles, and in a block alone 1.6 us.
constexpr int kClusterThreads = 1024;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterMax = 16;

// kAlone: a cluster of one block, with block barriers and plain addresses
template <int Items, bool kAlone>
__global__ void __launch_bounds__(kClusterThreads, 1)
k_sort_cluster(const uint64_t* __restrict__ keysIn, const uint32_t* __restrict__ valsIn, uint64_t* __restrict__ keysOut,
               uint32_t* __restrict__ valsOut, int n, int npass) {
    constexpr int kBlockKeys = kClusterThreads * Items;  // a power of two
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* skeys = reinterpret_cast<uint64_t*>(smem);
    uint32_t* svals = reinterpret_cast<uint32_t*>(skeys + kBlockKeys);
    uint32_t* warpHist = svals + kBlockKeys;                // [kClusterWarps][256]
    uint32_t* warpMask = warpHist + kClusterWarps * 256;    // [kClusterWarps][256]
    uint32_t* counts = warpMask + kClusterWarps * 256;      // [256]: this block's, read by the others
    uint32_t* start = counts + 256;                         // [256]: first position of this block's keys of a digit
    __shared__ uint32_t sums[8], quarter[4][256];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = kAlone ? 0 : (int)cluster.block_rank(), size = kAlone ? 1 : (int)cluster.num_blocks();
    auto sync = [&] {
        if (kAlone) __syncthreads();
        else cluster.sync();
    };
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int off0 = w * 32 * Items + lane;  // item k of this lane: position off0 + 32 k of the block
    const uint32_t lt = lanemask_lt();
    uint32_t* myHist = warpHist + w * 256;
    uint32_t* myMask = warpMask + w * 256;
    for (int i = lane; i < 256; i += 32) myMask[i] = 0u;
    // past the end: keys of the highest digit with the last positions; they
    // stay behind every key in every pass
    uint64_t key[Items];
    uint32_t val[Items];
#pragma unroll
    for (int k = 0; k < Items; k++) {
        const int i = rank * kBlockKeys + off0 + 32 * k;
        key[k] = i < n ? keysIn[i] : ~0ull;
        val[k] = i < n ? (valsIn ? valsIn[i] : (uint32_t)i) : 0u;
    }
    for (int pass = 0; pass < npass; pass++) {
        const int shift = 8 * pass;
        auto digit = [&](int k) { return (uint32_t)(key[k] >> shift) & 255u; };
        if (pass > 0) {
#pragma unroll
            for (int k = 0; k < Items; k++) {
                key[k] = skeys[off0 + 32 * k];
                val[k] = svals[off0 + 32 * k];
            }
        }
        for (int i = lane; i < 256; i += 32) myHist[i] = 0u;
        __syncwarp();
        uint32_t in[Items];  // rank among the warp's keys of the digit
#pragma unroll
        for (int k = 0; k < Items; k++) {
            const uint32_t d = digit(k);
            uint32_t peers = 0xffffffffu, before;
            if (__all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {
                before = myHist[d];
                __syncwarp();
                if (lane == 0) myHist[d] = before + 32u;
            } else {
                atomicOr(&myMask[d], 1u << lane);
                __syncwarp();
                peers = myMask[d];
                before = myHist[d];
                __syncwarp();
                if ((peers & lt) == 0u) {
                    myHist[d] = before + __popc(peers);
                    myMask[d] = 0u;
                }
            }
            in[k] = before + __popc(peers & lt);
            __syncwarp();
        }
        __syncthreads();
        {  // per digit: exclusive over the warps, a quarter of them per thread
            const int d = tid & 255, q = tid >> 8;
            uint32_t* h = warpHist + q * (kClusterWarps / 4) * 256 + d;
            uint32_t c[kClusterWarps / 4], s = 0;
#pragma unroll
            for (int k = 0; k < kClusterWarps / 4; k++) c[k] = h[k * 256];
#pragma unroll
            for (int k = 0; k < kClusterWarps / 4; k++) s += c[k];
            quarter[q][d] = s;
            __syncthreads();
            uint32_t at = 0;
#pragma unroll
            for (int k = 0; k < 3; k++) at += k < q ? quarter[k][d] : 0u;
            if (q == 3) counts[d] = at + s;
#pragma unroll
            for (int k = 0; k < kClusterWarps / 4; k++) {
                h[k * 256] = at;
                at += c[k];
            }
        }
        sync();  // all counts are there, and every block has its keys in registers
        if (tid < 256) {
            uint32_t before = 0, total = 0;
            if (kAlone) {
                total = counts[tid];
            } else {
                uint32_t c[kClusterMax];
#pragma unroll
                for (int b = 0; b < kClusterMax; b++) c[b] = b < size ? cluster.map_shared_rank(counts, b)[tid] : 0u;
#pragma unroll
                for (int b = 0; b < kClusterMax; b++) {
                    before += b < rank ? c[b] : 0u;
                    total += c[b];
                }
            }
            uint32_t x = total;  // scan over the digits
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) sums[w] = x;
            start[tid] = x - total + before;
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t x = start[tid];
            for (int k = 0; k < w; k++) x += sums[k];
            start[tid] = x;
        }
        __syncthreads();
        const bool last = pass == npass - 1;
#pragma unroll
        for (int k = 0; k < Items; k++) {
            const uint32_t d = digit(k);
            const uint32_t at = start[d] + myHist[d] + in[k];
            if (last) {
                if (at < (uint32_t)n) {
                    keysOut[at] = key[k];
                    valsOut[at] = val[k];
                }
            } else if (kAlone) {
                skeys[at] = key[k];
                svals[at] = val[k];
            } else {
                const int b = (int)(at / kBlockKeys);
                cluster.map_shared_rank(skeys, b)[at % kBlockKeys] = key[k];
                cluster.map_shared_rank(svals, b)[at % kBlockKeys] = val[k];
            }
        }
        sync();  // the keys have arrived (after the last pass: no block leaves while its counts are read)
    }
}

// ---------------------------------------------------------------- launchers
namespace {
size_t pass_smem() { return (size_t)kTile * (8 + 4) + (size_t)(kWarps * 256 + 3 * 256) * 4; }
size_t hist_smem(int npass) { return (size_t)npass * 256 * kHistCopies * 4; }
size_t cluster_smem(int items) {
    return (size_t)kClusterThreads * items * 12 + (size_t)(2 * kClusterWarps * 256 + 2 * 256) * 4;
}
template <int Items, bool kAlone>
cudaError_t cluster_init() {
    cudaError_t e = cudaFuncSetAttribute(k_sort_cluster<Items, kAlone>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)cluster_smem(Items));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_sort_cluster<Items, kAlone>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}
}  // namespace

int bh_sort_tile() { return kTile; }

cudaError_t bh_sort_init() {
    cudaError_t e = cudaFuncSetAttribute(k_sort_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pass_smem());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_sort_histogram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist_smem(8));
    if (e == cudaSuccess) e = cluster_init<1, true>();
    if (e == cudaSuccess) e = cluster_init<1, false>();
    if (e == cudaSuccess) e = cluster_init<2, false>();
    return e;
}

// The sizes where the cluster is the faster sort (8 passes of a standalone
// sort): 1,000 pairs 14.6 us against 39-48 by launches of tiles, 4,096 31 against
// 51, 16,384 (one key a thread) 41 against 56, 32,768 (two) 56 against 60; with
// four keys a thread 50,000 pairs take 92 against 61.  A GPU that cannot place
// clusters of 16 sorts by tiles.
int bh_sort_cluster_limit() {
    static const int limit = [] {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClusterMax);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = cluster_smem(2);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kClusterMax;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int fit = 0;
        if (bh_sort_init() != cudaSuccess || cudaOccupancyMaxActiveClusters(&fit, k_sort_cluster<2, false>, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            return 0;
        }
        return fit > 0 ? 2 * kClusterMax * kClusterThreads : 0;
    }();
    return limit;
}

cudaError_t bh_launch_sort_cluster(const uint64_t* keysIn, const uint32_t* valsIn, uint64_t* keysOut, uint32_t* valsOut,
                                   int n, int npass, cudaStream_t s) {
    const int items = n <= kClusterMax * kClusterThreads ? 1 : 2;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = cluster_smem(items);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[0].val.clusterDim.x = (unsigned)((n - 1) / (kClusterThreads * items) + 1);
    cfg.gridDim = dim3(attr[0].val.clusterDim.x);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto launch = [&](auto kernel) { return cudaLaunchKernelEx(&cfg, kernel, keysIn, valsIn, keysOut, valsOut, n, npass); };
    if (n <= kClusterThreads) return launch(k_sort_cluster<1, true>);
    return items == 1 ? launch(k_sort_cluster<1, false>) : launch(k_sort_cluster<2, false>);
}

cudaError_t bh_launch_sort_histogram(const uint64_t* keys, int n, uint32_t* hist, int npass, cudaStream_t s) {
    int grid = (n + kHistThreads * 8 - 1) / (kHistThreads * 8);
    const int cap = 3 * bh_sm_count();  // resident at once with 64 KB of counters each
    grid = grid < 1 ? 1 : (grid > cap ? cap : grid);
    k_sort_histogram<<<grid, kHistThreads, hist_smem(npass), s>>>(keys, n, hist, npass);
    return cudaGetLastError();
}

cudaError_t bh_launch_sort_pass(const uint64_t* keysIn, const uint32_t* valsIn, uint64_t* keysOut,
                                uint32_t* valsOut, int n, int shift, const uint32_t* hist,
                                uint32_t* status, int* tileCounter, int* err, int identityVals,
                                cudaStream_t s) {
    const int tiles = (n + kTile - 1) / kTile;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = pass_smem();
    cfg.stream = s;
    // passes after the first depend programmatically on their predecessor
    // (the first one follows the kernel that made its keys and histograms,
    // which its prologue reads)
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = shift > 0 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_sort_pass, keysIn, valsIn, keysOut, valsOut, n, shift, hist, status,
                              tileCounter, err, identityVals);
}

// Self-test of the bounded look-back wait: tile 1 looks back at a tile 0
// that never publishes; the wait gives up after BH_SPIN_LIMIT round trips,
// records BH_ERR_TIMEOUT and the kernel returns.
__global__ void k_lookback_selftest(const uint32_t* status, int* err) {
    if (threadIdx.x == 0) (void)lookback_exclusive(status, 1, 0, err);
}

cudaError_t bh_launch_lookback_selftest(const uint32_t* status, int* err, cudaStream_t s) {
    k_lookback_selftest<<<1, 32, 0, s>>>(status, err);
    return cudaGetLastError();
}

extern "C" int bh_selftest_bounded_wait(cudaStream_t s) {
    uint32_t* buf = nullptr;  // status words of two tiles (tile 0 left unpublished), then the error word
    const size_t words = 2 * 256 + 1;
    cudaError_t e = cudaMallocAsync(&buf, words * sizeof(uint32_t), s);
    if (e != cudaSuccess) return bh_note_cuda_error(e);
    int* err = reinterpret_cast<int*>(buf + 2 * 256);
    e = cudaMemsetAsync(buf, 0, words * sizeof(uint32_t), s);
    if (e == cudaSuccess) {
        k_lookback_selftest<<<1, 32, 0, s>>>(buf, err);
        e = cudaGetLastError();
    }
    int h = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaError_t f = cudaFreeAsync(buf, s);
    if (e == cudaSuccess) e = f;
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bh_note_cuda_error(e);
    return (h & BH_ERRBIT(BH_ERR_TIMEOUT)) ? BH_ERR_TIMEOUT : BH_OK;
}
