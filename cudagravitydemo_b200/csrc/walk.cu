// walk.cu — Barnes-Hut tree walk and kick-drift integrator (sm_100a).
//
// Semantics are the reference's calculateAcceleration (tree.cu:562-676):
// bodies are taken in groups of 32 Morton-consecutive bodies; starting from
// the root's children, a node is OPENED when it is not a leaf and at least one
// valid body of the group fails  size^2 < theta^2 * d^2  (size = x-extent /
// 2^level, d = distance from the body to the node's centre of mass,
// tree.cu:501-530, 610-634); otherwise every body of the group interacts with
// the node's monopole, Plummer-softened.  The set of interacting nodes is
// therefore a function of the group alone, and this kernel reproduces it
// exactly while changing how it is found:
//   - the 32 lanes test 64 different nodes per round, two each (the reference
//     tests one node per step with all 32 lanes);
//   - a node is accepted without a vote when the distance from its centre of
//     mass to the group's bounding box already satisfies the criterion with a
//     2^-16 relative margin (which dominates every rounding difference): 78%
//     of the nodes tested (1M disk);
//   - the others wait in a buffer until 32 are there.  Then each lane takes
//     one and opens it when a representative body (the group's body nearest
//     the box corner on the node's side) already fails the test; what is left
//     (9% of the nodes) waits in a second buffer for the exact group vote,
//     again 32 nodes at a time, one per lane, each lane running over the
//     group's bodies two at a time with packed FP32x2 arithmetic (same FP32
//     operations and order as the reference, so the decision is bit-identical);
//     opened nodes push their children;
//   - accepted nodes' (centre of mass, mass) are appended to a per-warp list
//     in shared memory and evaluated in bulk, two list entries per
//     instruction with sm_100's packed FP32x2 arithmetic: per pair of
//     interactions 3 SUB2, 3 FMA2, two MUFU rsqrt, 3 MUL2 and 3 FMA2, fed by
//     two 16-byte shared loads (the list is stored as four component arrays
//     x[], y[], z[], m[]: a 16-byte load yields two ready packed operands, and
//     appending consecutive entries stores without bank conflicts);
//   - sums are compensated per block of list entries (Kahan on the block
//     partials) when requested;
//   - warps fetch groups from an atomic cursor (dynamic load balance).
// What bounds it: instruction dispatch.  A packed FP32x2 instruction takes two
// dispatch cycles of a sub-partition, three when its three operands are
// distinct registers; counted so, dispatch is 94% busy (262K learned walk: 28.6K
// instructions and 13.3K packed second cycles per group in 47.8K cycles), 68% of it the
// evaluation at 15-16 cycles per 32 interactions (14 without register-port
// conflicts).  Everything that shortens the traversal's instruction stream
// therefore shows: waiting for full batches of 32 before the rarer, dearer
// tests (instead of running them, mostly empty, in every round) and explicit
// shared addresses took the 1M disk's walk from 1873 to 1647 us (learned, RMS
// 1e-3) and from 1587 to 1423 us (theta 0.5), and the 4M merger's step from
// 9.18 to 8.18 ms.
// Leaves never open, as in the reference (count <= 1 or no children).
// Extensions (template switches, off for the reference's semantics): the
// relative opening criterion with per-group budgets (the learned criterion),
// bucket leaves (an opened node with at most leafSize bodies contributes its
// bodies), and a group table for batches of independent systems.
#include <math.h>

#include "bh_internal.cuh"
#include "bh_kernels.cuh"

namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kThreads = kWarpsPerBlock * 32;
#ifndef BH_WALK_STACK_SMEM
#define BH_WALK_STACK_SMEM 768
#endif
#ifndef BH_WALK_LIST_CAP
#define BH_WALK_LIST_CAP 256
#endif
// stack entries per warp in shared memory when WalkArgs.stackSmem is 0; the
// size is a launch parameter (dynamic shared memory) that the autotuner sets
constexpr int kStackSmemDefault = BH_WALK_STACK_SMEM;
constexpr int kListCap = BH_WALK_LIST_CAP;      // interaction-list entries per warp (a multiple of 64)
#ifndef BH_WALK_MIN_BLOCKS_PLAIN
#define BH_WALK_MIN_BLOCKS_PLAIN 6
#endif
#ifndef BH_WALK_MIN_BLOCKS_RELATIVE
#define BH_WALK_MIN_BLOCKS_RELATIVE 6
#endif
#ifndef BH_WALK_MIN_BLOCKS_WIDE
#define BH_WALK_MIN_BLOCKS_WIDE 4
#endif
// Resident blocks per SM the register allocation must allow (64K registers /
// (128 threads x blocks)): fewer blocks, more registers per thread.  Measured
// on the 1M disk, the walk is faster with registers than with warps: 6 blocks
// (80 registers), which is also what shared memory allows with the 256-entry
// list and the default 768-entry stack (38 KB per block): 1652 us learned, 1432
// plain; 7 blocks (72 registers, 512-entry stack) 1751 and 1465, 8 blocks (64
// registers) 1806 and 1577, 5 blocks (96 registers) 1668 and 1451.
constexpr int kMinBlocksPlain = BH_WALK_MIN_BLOCKS_PLAIN;
constexpr int kMinBlocksRelative = BH_WALK_MIN_BLOCKS_RELATIVE;
// 64-body groups (two bodies per lane), every criterion: 4 blocks (up to 128
// registers; 110 used) measured 7% faster than 6 blocks with spills
constexpr int kMinBlocksWide = BH_WALK_MIN_BLOCKS_WIDE;
// Few 32-body groups: the time is one long group's chain of rounds, and warps in
// other slots hide nothing.  More registers (3 blocks, up to 168; 138 to 150 used)
// let one warp overlap its own entries: a list of 224 takes 3,650 cycles instead
// of 7,550 (the dispatch port alone needs 3,600), a vote unrolled whole 1,120 instead of
// 1,500.  Walk before and after, us, theta 0.5 Plummer spheres unless said: 1,000
// bodies 42 and 39, 4,000 76 and 66, 16,384 92 and 80, 36,000 145 and 133, 60,000
// 170 and 164, 100,000 203 and 195; disks of 80,000 171 and 145, learned of 100,000
// 203 and 183.  Beyond that throughput counts again: 125,000 225 and 232 (a disk 211
// and 199), 150,000 254 and 268, 262,144 learned 416 and 444.  The line is drawn
// at 24 groups per SM (113,000 bodies).  Blocks of 2 and 4 per SM were the same up
// to 36,000 bodies, 226 and 187 us at 100,000, 151 and 169 at the disk of 80,000;
// prefetching the children of opened nodes into L1 gave nothing (80 to 82 us at
// 16,384), and evaluators in warps of their own beside the walker gave less (82).
constexpr int kMinBlocksFew = 3;
constexpr int kFewGroupsPerSm = 24;
__host__ __device__ constexpr int walk_min_blocks(bool relative, bool wide, bool few) {
    return few ? kMinBlocksFew : wide ? kMinBlocksWide : (relative ? kMinBlocksRelative : kMinBlocksPlain);
}
constexpr int kBlocksPerSm = 8;  // persistent grid: blocks launched per SM (the excess waits)
constexpr int kSpillPerWarp = 4096;  // global stack entries per warp beyond shared memory
constexpr float kBoxMargin = 1.0f - 1.0f / 65536.0f;
// nodes waiting for their representative test (fewer than 32 before a round
// of 64 box tests) and for the exact vote (fewer than 32 before 32 more)
constexpr int kPendCap = 96;
constexpr int kVoteCap = 64;

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two floats packed in one 64-bit register (low half = first), and the
// sm_100 packed FP32x2 operations on them (round to nearest).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// min of three, for a squared distance against a bound: a NaN stays one (the
// comparison with it then opens), or is passed over
__device__ __forceinline__ float min3_nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Shared memory by 32-bit address: one base register per warp and immediate
// offsets.  (Through C++ arrays the compiler kept recomputing the thread's
// indices and the window's base in every round.)
__device__ __forceinline__ int lds_i(unsigned a) {
    int v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float lds_f(unsigned a) { return __int_as_float(lds_i(a)); }
__device__ __forceinline__ float4 lds_f4(unsigned a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ ulonglong2 lds_2x2(unsigned a) {  // two packed pairs
    ulonglong2 v;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts_i(unsigned a, int v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v)); }
__device__ __forceinline__ void sts_f(unsigned a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v)); }
__device__ __forceinline__ void sts_f4(unsigned a, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
}
// The lanes meet.  Volatile as the accesses above, which name no memory: the
// compiler keeps all of them in order.
__device__ __forceinline__ void sync_warp() { asm volatile("bar.warp.sync 0xffffffff;" ::: "memory"); }

// A warp's shared memory, byte offsets from its base:
//   list   the interaction list as four arrays of kListCap floats: x[], y[], z[], m[]
//   body   the group's bodies for the exact vote, in pairs: (x0, x1, y0, y1),
//          (z0, z1, k0, k1), k the body's share of the relative criterion; a
//          partial group is filled up with copies of its first body, which
//          change no verdict
//   rep    the group's representative body of each box octant, (x, y, z, k)
//   sum    per lane: running sums x, y, z, compensations x, y, z (then the
//          second body's): touched once per flushed list block only, and the
//          registers they free let more warps be resident
//   pend   nodes the box test could not accept, and
//   vote   of those the ones no representative body opens
//   group  the group being walked and its interaction-list length so far
//   stack  the traversal stack's first stackSmem entries
template <bool kWide>
struct WarpMem {
    static constexpr unsigned list = 0, listArray = 4u * kListCap;
    static constexpr unsigned body = list + 4 * listArray;
    static constexpr unsigned rep = body + 16u * (kWide ? 64 : 32);
    static constexpr unsigned sum = rep + 16u * 8;
    static constexpr unsigned pend = sum + 128u * (kWide ? 12 : 6);
    static constexpr unsigned vote = pend + 4u * kPendCap;
    static constexpr unsigned group = vote + 4u * kVoteCap;
    static constexpr unsigned stack = group + 16;
    static constexpr unsigned bytes(int stackSmem) { return stack + 4u * (unsigned)stackSmem; }
};

// The reference's d^2 (tree.cu:611) as its compiled walk evaluates it:
// fma(dz, dz, fma(dx, dx, dy * dy)).  The opening test must round exactly
// like the reference's for the interaction sets to be identical.
__device__ __forceinline__ float ref_dist_sq(float dx, float dy, float dz) {
    return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

}  // namespace

// One warp per group of 32 bodies (kWide: 64, two per lane).  kFew: the same walk
// compiled for latency, bit-identical.
template <bool kFused, bool kCompensated, bool kRelative, bool kBuckets, bool kWide, bool kFew>
__global__ void __launch_bounds__(kThreads, walk_min_blocks(kRelative, kWide, kFew))
k_walk(const WalkArgs a) {
    constexpr int kW = kWide ? 64 : 32;
    const float4* __restrict__ pos = a.pos;
    const WalkNode* __restrict__ wn = a.wn;
    const int n = a.n;
    const float eps2 = a.eps2, G = a.G, dt = a.dt;
    int* err = a.err;
    const int spillPerWarp = kSpillPerWarp;
    const int stackSmem = a.stackSmem;
    using Mem = WarpMem<kWide>;
    constexpr unsigned kSums = kWide ? 12 : 6;
    extern __shared__ __align__(16) char sDyn[];
    int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    unsigned lt = lanemask_lt(), sm = (unsigned)__cvta_generic_to_shared(sDyn) + wi * Mem::bytes(stackSmem);
    // (opaque from here on: kept in registers, not recomputed in every round)
    asm volatile("" : "+r"(lane), "+r"(lt), "+r"(sm));
    const unsigned sl = sm + 4u * lane;  // this lane's column
    int* spill = a.spill + (size_t)(blockIdx.x * kWarpsPerBlock + wi) * spillPerWarp;
    const int stackCap = stackSmem + spillPerWarp;
    const int groups = a.groupTable ? a.groups : (n + kW - 1) / kW;
    const int leafSize = a.leafSize > 1 ? a.leafSize : 1;  // nodes with at most this many bodies are buckets
    unsigned nInteract = 0, nTested = 0, nVote = 0;
    // interactions of this warp so far; handed to the 64-bit total before the
    // 32-bit count could wrap (uniform across the warp)
    auto countInteractions = [&](int len, int nValid) {
        nInteract += (unsigned)len * (unsigned)nValid;
        if (nInteract >= 0x80000000u) {
            if (lane == 0) atomicAdd(&a.ctr->interactions, (unsigned long long)nInteract);
            nInteract = 0;
        }
    };
    int maxTop = 0;

    for (;;) {
        int g = 0;
        if (lane == 0) {
            g = atomicAdd(&a.ctr->groupCursor, 1);
            if (a.groupOrder && g < groups) g = a.groupOrder[g];  // longest lists first
        }
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= groups) break;
        // the group's bodies and the root of its tree (a batch: one per system)
        int first, cnt, root = 0;
        if (a.groupTable) {
            const int4 gt = a.groupTable[g];
            first = gt.x;
            cnt = gt.y;
            root = gt.z;
        } else {
            first = g * kW;
            cnt = n - first < kW ? n - first : kW;
        }
        const int b = first + lane;
        const bool valid = lane < cnt;
        const float4 p = valid ? pos[b] : make_float4(0.f, 0.f, 0.f, 0.f);
        // the second body of the lane (64-body groups)
        const int b1 = b + 32;
        const bool valid1 = kWide && lane + 32 < cnt;
        float3 p1 = make_float3(0.f, 0.f, 0.f);
        if (kWide && valid1) {
            const float4 q = pos[b1];
            p1 = make_float3(q.x, q.y, q.z);
        }
        const int nValid = cnt;
        // opening parameters of this group (per 32-body group; a 64-body group
        // takes the smaller theta and budget of its two halves)
        float theta = a.theta, kA = 0.f;
        if (a.groupParam) {
            float2 gp = a.groupParam[kWide ? 2 * g : g];
            if (kWide && 2 * g + 1 < a.groupParamCount) {
                const float2 q = a.groupParam[2 * g + 1];
                gp.x = fminf(gp.x, q.x);
                gp.y = fminf(gp.y, q.y);
            }
            theta = gp.x;
            kA = gp.y / G;
        } else {
            kA = a.alpha / G;
        }
        const float thetaSq = __fmul_rn(theta, theta);
        const float thetaSqBox = thetaSq * kBoxMargin;
        // relative criterion: open when M s^2 > kA |a_b| d^4 for some body
        float myA = 0.f, myA1 = 0.f, kAmin = 0.f;
        if (kRelative) {
            myA = valid ? a.aMagIn[b] : INFINITY;
            float aMin = myA;
            if (kWide) {
                myA1 = valid1 ? a.aMagIn[b1] : INFINITY;
                aMin = fminf(aMin, myA1);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) aMin = fminf(aMin, __shfl_xor_sync(0xffffffffu, aMin, o));
            kAmin = kA * aMin * kBoxMargin;
        }
        {  // the bodies as the vote reads them
            const float4 f = make_float4(__shfl_sync(0xffffffffu, p.x, 0), __shfl_sync(0xffffffffu, p.y, 0),
                                         __shfl_sync(0xffffffffu, p.z, 0), __shfl_sync(0xffffffffu, myA, 0));
            auto put = [&](int i, bool v, float x, float y, float z, float am) {
                const unsigned e = sm + Mem::body + 32u * (i >> 1) + 4u * (i & 1);
                sts_f(e, v ? x : f.x);
                sts_f(e + 8, v ? y : f.y);
                sts_f(e + 16, v ? z : f.z);
                sts_f(e + 24, kRelative ? kA * (v ? am : f.w) : 0.f);
            };
            put(lane, valid, p.x, p.y, p.z, myA);
            if (kWide) put(lane + 32, valid1, p1.x, p1.y, p1.z, myA1);
        }

        // group box as centre +- half extent; the half extent is rounded
        // outward so the box contains every body of the group exactly
        float bm[3], be[3];
        {
            float lo[3] = {valid ? p.x : INFINITY, valid ? p.y : INFINITY, valid ? p.z : INFINITY};
            float hi[3] = {valid ? p.x : -INFINITY, valid ? p.y : -INFINITY, valid ? p.z : -INFINITY};
            if (kWide && valid1) {
                lo[0] = fminf(lo[0], p1.x); lo[1] = fminf(lo[1], p1.y); lo[2] = fminf(lo[2], p1.z);
                hi[0] = fmaxf(hi[0], p1.x); hi[1] = fmaxf(hi[1], p1.y); hi[2] = fmaxf(hi[2], p1.z);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
                    hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
                }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                bm[k] = 0.5f * (lo[k] + hi[k]);
                const float mag = fmaxf(fabsf(lo[k]), fabsf(hi[k]));
                be[k] = __fmul_ru(0.5f, __fsub_ru(hi[k], lo[k])) + mag * 1.0e-6f;
            }
        }
        // representative bodies, one per octant of the group box: the valid
        // body nearest each corner of the box (among bodies whose squared
        // distances agree to 32 ulps, any).  A node is tested against the
        // representative of the octant its centre of mass lies in — a body on
        // the node's side of the group, so that a node some body fails is
        // mostly found without a vote (a third fewer votes than with the body
        // nearest the centre)
        {
#pragma unroll
            for (int o = 0; o < 8; o++) {
                const float cx = (o & 4) ? bm[0] + be[0] : bm[0] - be[0];
                const float cy = (o & 2) ? bm[1] + be[1] : bm[1] - be[1];
                const float cz = (o & 1) ? bm[2] + be[2] : bm[2] - be[2];
                float d = valid ? (p.x - cx) * (p.x - cx) + (p.y - cy) * (p.y - cy) + (p.z - cz) * (p.z - cz)
                                : INFINITY;
                bool second = false;
                if (kWide && valid1) {
                    const float d1 = (p1.x - cx) * (p1.x - cx) + (p1.y - cy) * (p1.y - cy) + (p1.z - cz) * (p1.z - cz);
                    if (d1 < d) { d = d1; second = true; }
                }
                const unsigned best = __reduce_min_sync(0xffffffffu, (__float_as_uint(d) & ~31u) | (unsigned)lane);
                if ((best & 31u) == (unsigned)lane)
                    sts_f4(sm + Mem::rep + 16u * o, second ? make_float4(p1.x, p1.y, p1.z, kA * myA1)
                                                           : make_float4(p.x, p.y, p.z, kA * myA));
            }
        }

        // root's children onto the stack
        int top;
        {
            const int rb = wn[root].childBegin, re = wn[root].childEnd;
            top = re - rb;
            if (lane < top) sts_i(sl + Mem::stack, rb + lane);
        }
        int listLen = 0, pendLen = 0, voteLen = 0;
        if (lane == 0) {
            sts_i(sm + Mem::group, g);
            sts_i(sm + Mem::group + 4, 0);
        }
#pragma unroll
        for (unsigned k = 0; k < kSums; k++) sts_f(sl + Mem::sum + 128u * k, 0.f);  // this lane's column only
        sync_warp();

        // interactions with list entries [0, cnt); partial sums Kahan-added
        auto kahan = [&](float ax, float ay, float az, unsigned S) {
            float s0 = lds_f(S), s1 = lds_f(S + 128), s2 = lds_f(S + 256);
            if (kCompensated) {
                float c0 = lds_f(S + 384), c1 = lds_f(S + 512), c2 = lds_f(S + 640);
                float y, t;
                y = ax - c0; t = s0 + y; c0 = (t - s0) - y; s0 = t;
                y = ay - c1; t = s1 + y; c1 = (t - s1) - y; s1 = t;
                y = az - c2; t = s2 + y; c2 = (t - s2) - y; s2 = t;
                sts_f(S + 384, c0);
                sts_f(S + 512, c1);
                sts_f(S + 640, c2);
            } else {
                s0 += ax; s1 += ay; s2 += az;
            }
            sts_f(S, s0);
            sts_f(S + 128, s1);
            sts_f(S + 256, s2);
        };
        auto flush = [&](int cnt) {
            float ax, ay, az;
            float bx = 0.f, by = 0.f, bz = 0.f;  // second body (64-body groups)
            // one 16-byte load of a component array gives four entries' x,
            // i.e. two packed pairs
            const f32x2 px2 = pack2(p.x, p.x), py2 = pack2(p.y, p.y), pz2 = pack2(p.z, p.z);
            const f32x2 qx2 = pack2(p1.x, p1.x), qy2 = pack2(p1.y, p1.y), qz2 = pack2(p1.z, p1.z);
            const f32x2 e2 = pack2(eps2, eps2);
            const unsigned end = sm + 4u * cnt;  // cnt is a multiple of 32
            f32x2 ax2 = 0ull, ay2 = 0ull, az2 = 0ull;
            f32x2 bx2 = 0ull, by2 = 0ull, bz2 = 0ull;
            // one packed body-pair interaction: (bx, by, bz) against two entries
            auto pair = [&](f32x2 ex, f32x2 ey, f32x2 ez, f32x2 em, f32x2 ox, f32x2 oy, f32x2 oz, f32x2& sx2,
                            f32x2& sy2, f32x2& sz2) {
                const f32x2 dx = sub2(ex, ox), dy = sub2(ey, oy), dz = sub2(ez, oz);
                f32x2 r2 = fma2(dx, dx, e2);
                r2 = fma2(dy, dy, r2);
                r2 = fma2(dz, dz, r2);
                float r2a, r2b;
                unpack2(r2, r2a, r2b);
                const f32x2 ri = pack2(rsqrt_approx(r2a), rsqrt_approx(r2b));
                const f32x2 f = mul2(mul2(em, ri), mul2(ri, ri));
                sx2 = fma2(f, dx, sx2);
                sy2 = fma2(f, dy, sy2);
                sz2 = fma2(f, dz, sz2);
            };
            auto quad = [&](unsigned L) {  // four list entries
                const ulonglong2 x = lds_2x2(L), y = lds_2x2(L + Mem::listArray);
                const ulonglong2 z = lds_2x2(L + 2 * Mem::listArray), m = lds_2x2(L + 3 * Mem::listArray);
                pair(x.x, y.x, z.x, m.x, px2, py2, pz2, ax2, ay2, az2);
                if (kWide) pair(x.x, y.x, z.x, m.x, qx2, qy2, qz2, bx2, by2, bz2);
                pair(x.y, y.y, z.y, m.y, px2, py2, pz2, ax2, ay2, az2);
                if (kWide) pair(x.y, y.y, z.y, m.y, qx2, qy2, qz2, bx2, by2, bz2);
            };
            constexpr unsigned kQuads = kWide ? 2 : 8;
#pragma unroll 1
            for (unsigned L = sm; L < end; L += 16 * kQuads)
#pragma unroll
                for (unsigned k = 0; k < kQuads; k++) quad(L + 16 * k);
            float a0, a1;
            unpack2(ax2, a0, a1);
            ax = a0 + a1;
            unpack2(ay2, a0, a1);
            ay = a0 + a1;
            unpack2(az2, a0, a1);
            az = a0 + a1;
            if (kWide) {
                unpack2(bx2, a0, a1);
                bx = a0 + a1;
                unpack2(by2, a0, a1);
                by = a0 + a1;
                unpack2(bz2, a0, a1);
                bz = a0 + a1;
            }
            kahan(ax, ay, az, sl + Mem::sum);
            if (kWide) kahan(bx, by, bz, sl + Mem::sum + 128u * (kSums - 6));
        };

        // A stack entry is a node index (>= 0) or, below a bucket node that
        // was opened, a body b encoded as -(b + 2): a body is a leaf, always
        // accepted.
        auto popped = [&](int at) -> int {
            return at < stackSmem ? lds_i(sm + Mem::stack + 4u * at) : spill[at - stackSmem];
        };
        auto append = [&](const float4& com, bool accept, int k) {
            if (!accept) return;  // component arrays: consecutive entries, conflict-free stores
            const unsigned L = sm + 4u * k;
            sts_f(L, com.x);
            sts_f(L + Mem::listArray, com.y);
            sts_f(L + 2 * Mem::listArray, com.z);
            sts_f(L + 3 * Mem::listArray, com.w);
        };
        // The box test of one stack entry: true when it is a leaf, a body or
        // far enough from the whole group, false when it needs a closer look.
        auto closed = [&](int idx, float4& com) -> bool {
            const int li = kBuckets && idx < 0 ? 0 : idx;
            com = wn[li].com;
            const int4 meta = *reinterpret_cast<const int4*>(&wn[li].childBegin);
            if (kBuckets && idx < 0) com = pos[-idx - 2];
            const float gx = fmaxf(fabsf(com.x - bm[0]) - be[0], 0.f);
            const float gy = fmaxf(fabsf(com.y - bm[1]) - be[1], 0.f);
            const float gz = fmaxf(fabsf(com.z - bm[2]) - be[2], 0.f);
            const float D2 = gx * gx + gy * gy + gz * gz;
            const float sizeSq = __int_as_float(meta.z);
            bool c = thetaSqBox * D2 > sizeSq;
            if (kRelative) c = c & (com.w * sizeSq < kAmin * (D2 * D2));
            c = c | (meta.x == meta.y);  // a leaf never opens
            if (kBuckets) c = c | (idx < 0);
            return c;
        };

        bool overflow = false;
        for (;;) {
            // (a round of fewer than 32 entries waits until nothing else is
            // left to do: 152 against 157 us at 16,384 bodies, large walks the same)
            if ((top >= 32 || (top > 0 && (pendLen | voteLen) == 0)) && (pendLen | voteLen) < 32) {
                // ---- box tests of up to 64 stack entries, two per lane
                const int take = top < 64 ? top : 64;
                top -= take;
                const bool h0 = lane < take, h1 = lane + 32 < take;
                int i0 = 0, i1 = 0;
                if (top + 64 <= stackSmem) {  // uniform: the usual case
                    const unsigned q = sl + Mem::stack + 4u * top;
                    i0 = lds_i(q);
                    i1 = lds_i(q + 128);
                    i0 = h0 ? i0 : 0;
                    i1 = h1 ? i1 : 0;
                } else {
                    if (h0) i0 = popped(top + lane);
                    if (h1) i1 = popped(top + 32 + lane);
                }
                float4 c0, c1;
                const bool cl0 = closed(i0, c0), cl1 = closed(i1, c1);
                const bool acc0 = h0 & cl0, acc1 = h1 & cl1, pe0 = h0 & !cl0, pe1 = h1 & !cl1;
                const unsigned am0 = __ballot_sync(0xffffffffu, acc0), am1 = __ballot_sync(0xffffffffu, acc1);
                // (every entry below an entry that is pending is either
                // accepted or pending: the ranks of the one give the other's)
                const int r0 = __popc(am0 & lt), r1 = __popc(am1 & lt), n0 = __popc(am0), n1 = __popc(am1);
                const int k0 = (take < 32 ? take : 32) - n0;
                append(c0, acc0, listLen + r0);
                append(c1, acc1, listLen + n0 + r1);
                if (pe0) sts_i(sl + Mem::pend + 4u * (pendLen - r0), i0);
                if (pe1) sts_i(sl + Mem::pend + 4u * (pendLen + k0 - r1), i1);
                listLen += n0 + n1;
                pendLen += take - n0 - n1;
                nTested += take;
            } else {
                // ---- 32 pending nodes (fewer once the stack is empty), one
                // per lane: against a representative body, or by the exact vote
                const bool vote = voteLen >= 32 || pendLen == 0;
                int len = vote ? voteLen : pendLen;
                if (len == 0) break;
                const int take = len < 32 ? len : 32;
                len -= take;
                const bool has = lane < take;
                int idx = 0;
                if (has) idx = lds_i(sl + (vote ? Mem::vote : Mem::pend) + 4u * len);
                if (vote) voteLen = len;
                else pendLen = len;
                const float4 com = wn[idx].com;
                const int4 meta = *reinterpret_cast<const int4*>(&wn[idx].childBegin);
                const float sizeSq = __int_as_float(meta.z);
                const float ms = com.w * sizeSq;
                bool open = false;
                if (vote) {
                    // the reference's group vote (tree.cu:629-640): open when
                    // any body of the group fails; two bodies per pass, every
                    // packed operation rounding like the scalar one
                    const f32x2 nx = pack2(com.x, com.x), ny = pack2(com.y, com.y), nz = pack2(com.z, com.z);
                    const f32x2 th2 = pack2(thetaSq, thetaSq);
                    // any body fails: the nearest does (rounding is monotonic)
                    float tMin = INFINITY, rMin = INFINITY;
#pragma unroll(kFew ? 16 : 4)  // (16 in every walk: 1% slower with 6 blocks' registers)
                    for (unsigned B = sm + Mem::body; B < sm + Mem::body + 16u * kW; B += 32) {
                        const ulonglong2 xy = lds_2x2(B), zk = lds_2x2(B + 16);
                        const f32x2 dx = sub2(xy.x, nx), dy = sub2(xy.y, ny), dz = sub2(zk.x, nz);
                        const f32x2 d2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));  // ref_dist_sq, packed
                        float ta, tb;
                        unpack2(mul2(th2, d2), ta, tb);
                        tMin = min3_nan(tMin, ta, tb);
                        if (kRelative) {
                            float ra, rb;
                            unpack2(mul2(zk.y, mul2(d2, d2)), ra, rb);
                            rMin = min3(rMin, ra, rb);
                        }
                    }
                    open = !(sizeSq < tMin);
                    if (kRelative) open = open | (ms > rMin);
                    open = open & has;
                    const bool acc = has & !open;
                    const unsigned am = __ballot_sync(0xffffffffu, acc);
                    append(com, acc, listLen + __popc(am & lt));
                    listLen += __popc(am);
                    nVote += take;
                } else {
                    const int oc = (com.x > bm[0] ? 4 : 0) | (com.y > bm[1] ? 2 : 0) | (com.z > bm[2] ? 1 : 0);
                    const float4 r = lds_f4(sm + Mem::rep + 16u * oc);  // (x, y, z, kA |a|) of the octant's representative
                    const float d2 = ref_dist_sq(r.x - com.x, r.y - com.y, r.z - com.z);
                    open = !(sizeSq < __fmul_rn(thetaSq, d2));
                    if (kRelative) open = open | (ms > r.w * (d2 * d2));
                    open = open & has;
                    const bool un = has & !open;
                    const unsigned um = __ballot_sync(0xffffffffu, un);
                    if (un) sts_i(sm + Mem::vote + 4u * (voteLen + __popc(um & lt)), idx);
                    voteLen += __popc(um);
                }
                // opened nodes -> their children (next level, at most 8;
                // anything else is a broken tree, reported rather than
                // followed) or, for a bucket (at most leafSize bodies), its
                // bodies: entries f + d * c, c < cnt
                int f = meta.x, d = 1, c = 0;
                if (open) {
                    c = meta.y - meta.x;
                    if (kBuckets && meta.w <= leafSize) {
                        f = -(a.nFirst[idx] + 2);
                        d = -1;
                        c = meta.w;
                    } else if (meta.x <= idx || c > 8) {
                        bh_set_error(err, BH_ERR_INTERNAL);
                        c = 0;
                    }
                }
                int incl = c, pushed;
                if (kFew && !kBuckets) {
                    // c <= 8: bit by bit, four ballots at once instead of a chain of
                    // shuffles (1.5% of a small walk; at 1M bodies 0.3% slower, it
                    // is more instructions)
                    const unsigned w0 = __ballot_sync(0xffffffffu, c & 1), w1 = __ballot_sync(0xffffffffu, c & 2);
                    const unsigned w2 = __ballot_sync(0xffffffffu, c & 4), w3 = __ballot_sync(0xffffffffu, c & 8);
                    incl += __popc(w0 & lt) + 2 * __popc(w1 & lt) + 4 * __popc(w2 & lt) + 8 * __popc(w3 & lt);
                    pushed = __popc(w0) + 2 * __popc(w1) + 4 * __popc(w2) + 8 * __popc(w3);
                } else {
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += y;
                    }
                    pushed = __shfl_sync(0xffffffffu, incl, 31);
                }
                if (top + pushed > stackCap) {
                    overflow = true;
                    break;
                }
                const int base = top + incl - c;
                if (top + pushed <= stackSmem) {  // uniform: the usual case
                    const unsigned q = sm + Mem::stack + 4u * base;
                    if (kBuckets && leafSize > 8) {
                        const int most = __reduce_max_sync(0xffffffffu, c);
                        for (int k = 0; k < most; k++)
                            if (k < c) sts_i(q + 4u * k, f + d * k);
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; k++)  // predicated, no loop
                            if (k < c) sts_i(q + 4u * k, kBuckets ? f + d * k : f + k);
                    }
                } else {
                    for (int k = 0; k < c; k++) {
                        const int at = base + k, v = f + d * k;
                        if (at < stackSmem) sts_i(sm + Mem::stack + 4u * at, v);
                        else spill[at - stackSmem] = v;
                    }
                }
                top += pushed;
                maxTop = top > maxTop ? top : maxTop;
            }
            sync_warp();
            if (listLen > kListCap - 64) {
                // the whole blocks of 32 entries; what is left moves to the front
                const int whole = listLen & ~31;
                flush(whole);
                countInteractions(whole, nValid);
                if (lane == 0) sts_i(sm + Mem::group + 4, lds_i(sm + Mem::group + 4) + whole);
                listLen -= whole;
                const bool left = lane < listLen;
                const unsigned L = left ? sl + 4u * whole : sm;
                const float4 e = make_float4(lds_f(L), lds_f(L + Mem::listArray), lds_f(L + 2 * Mem::listArray),
                                             lds_f(L + 3 * Mem::listArray));
                sync_warp();
                append(e, left, lane);
                sync_warp();
            }
        }
        if (overflow && lane == 0) bh_set_error(err, BH_ERR_STACK_OVERFLOW);
        sync_warp();  // (an overflow left its round after other lanes' entries were appended)
        if (listLen > 0) {
            // the last block, filled up with massless copies of its last entry
            // (they add zero wherever that entry's own term is finite)
            const int whole = (listLen + 31) & ~31;
            const unsigned L = sm + 4u * (listLen - 1);
            append(make_float4(lds_f(L), lds_f(L + Mem::listArray), lds_f(L + 2 * Mem::listArray), 0.f),
                   listLen + lane < whole, listLen + lane);
            sync_warp();
            flush(whole);
            countInteractions(listLen, nValid);
            if (lane == 0) sts_i(sm + Mem::group + 4, lds_i(sm + Mem::group + 4) + listLen);
        }
        if (a.groupLen && lane == 0) a.groupLen[lds_i(sm + Mem::group)] = lds_i(sm + Mem::group + 4);
        sync_warp();
        // results of one body: acceleration, |a|, and the fused kick-drift
        auto finish = [&](int bi, float bx, float by, float bz, float bm_, unsigned S) {
            float gx = lds_f(S), gy = lds_f(S + 128), gz = lds_f(S + 256);
            if (kCompensated) {
                gx -= lds_f(S + 384);
                gy -= lds_f(S + 512);
                gz -= lds_f(S + 640);
            }
            gx *= G; gy *= G; gz *= G;
            if (a.accOut) a.accOut[bi] = make_float3(gx, gy, gz);
            if (a.aMagOut) a.aMagOut[bi] = sqrtf(gx * gx + gy * gy + gz * gz);
            if (kFused) {
                // tree.cu:694-702: v = v + a dt, x = x + v dt (both fused)
                const float3 v = a.velIn[bi];
                const float vx = __fmaf_rn(gx, dt, v.x), vy = __fmaf_rn(gy, dt, v.y), vz = __fmaf_rn(gz, dt, v.z);
                a.velOut[bi] = make_float3(vx, vy, vz);
                const float4 np = make_float4(__fmaf_rn(vx, dt, bx), __fmaf_rn(vy, dt, by), __fmaf_rn(vz, dt, bz), bm_);
                a.posOut[bi] = np;
                if (a.idOut) a.idOut[bi] = a.idIn[bi];
                if (a.posHost) {  // the caller's host arrays, written over PCIe as groups finish
                    a.posHost[bi] = np;
                    a.velHost[bi] = make_float3(vx, vy, vz);
                    a.idHost[bi] = a.idIn[bi];
                }
            }
        };
        if (valid) finish(b, p.x, p.y, p.z, p.w, sl + Mem::sum);
        if (kWide && valid1) finish(b1, p1.x, p1.y, p1.z, pos[b1].w, sl + Mem::sum + 128u * (kSums - 6));
    }
    if (lane == 0) {
        atomicAdd(&a.ctr->interactions, (unsigned long long)nInteract);
        atomicAdd(&a.ctr->nodesTested, (unsigned long long)nTested);
        atomicAdd(&a.ctr->undecided, (unsigned long long)nVote);
        atomicMax(&a.ctr->maxStack, maxTop);
    }
}

// Walk order for the next walk: the groups by decreasing interaction-list
// length of the last walk (a group covers almost the same bodies from one
// step to the next), so that the persistent grid's warps finish together
// instead of waiting on a few long groups taken last.  A counting sort on 64
// logarithmic length bins in two launches of one thread per group: per-block
// bin counts, then each block finds where its groups of each bin start and
// scatters them.  The order inside a bin is arbitrary (it changes only which
// warp walks a group, never a result).
constexpr int kOrderThreads = 1024;
constexpr int kOrderBins = 64;

__device__ __forceinline__ int order_bin(int l) {
    l = l < 0 ? 0 : (l > (1 << 15) ? (1 << 15) : l);
    const int b = (int)(4.0f * __log2f((float)l + 1.0f));  // 4 bins per doubling
    return kOrderBins - 1 - (b < kOrderBins - 1 ? b : kOrderBins - 1);  // longest first
}

// blockHist[block][bin] = groups of this block's 1024 in each bin
__global__ void __launch_bounds__(kOrderThreads) k_group_order_count(const int* __restrict__ len, int groups,
                                                                     int* __restrict__ blockHist) {
    __shared__ int hist[kOrderBins];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < kOrderBins) hist[threadIdx.x] = 0;
    __syncthreads();
    const int g = blockIdx.x * kOrderThreads + threadIdx.x;
    const int b = g < groups ? order_bin(len[g]) : -1;
    // neighbouring groups have similar lengths: one atomic per bin and warp
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    if (b >= 0 && lane == __ffs(peers) - 1) atomicAdd(&hist[b], __popc(peers));
    __syncthreads();
    if (threadIdx.x < kOrderBins) blockHist[blockIdx.x * kOrderBins + threadIdx.x] = hist[threadIdx.x];
}

// order[pos] = g, pos = (groups in longer bins) + (groups of this bin in
// earlier blocks) + rank in this block
__global__ void __launch_bounds__(kOrderThreads) k_group_order_scatter(const int* __restrict__ len, int groups,
                                                                       const int* __restrict__ blockHist,
                                                                       int* __restrict__ order) {
    __shared__ int base[kOrderBins];
    __shared__ int firstHalf;  // groups in bins 0..31 (all blocks)
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < kOrderBins) {  // two warps, 32 bins each
        int total = 0, before = 0;
        for (int k = 0; k < (int)gridDim.x; k++) {
            const int c = blockHist[k * kOrderBins + threadIdx.x];
            total += c;
            if (k < (int)blockIdx.x) before += c;
        }
        int x = total;  // inclusive scan of the bin totals within the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        base[threadIdx.x] = x - total + before;
        if (threadIdx.x == 31) firstHalf = x;
    }
    __syncthreads();
    if (threadIdx.x >= 32 && threadIdx.x < kOrderBins) base[threadIdx.x] += firstHalf;
    __syncthreads();
    const int g = blockIdx.x * kOrderThreads + threadIdx.x;
    const int b = g < groups ? order_bin(len[g]) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    const int leader = __ffs(peers) - 1;
    int at = 0;
    if (b >= 0 && lane == leader) at = atomicAdd(&base[b], __popc(peers));
    at = __shfl_sync(0xffffffffu, at, leader);
    if (b >= 0) order[at + __popc(peers & lanemask_lt())] = g;
}

int bh_group_order_hist_ints(int groups) { return ((groups + kOrderThreads - 1) / kOrderThreads) * kOrderBins; }

cudaError_t bh_launch_group_order(const int* len, int groups, int* order, int* blockHist, cudaStream_t s) {
    if (groups <= 0) return cudaSuccess;
    const int blocks = (groups + kOrderThreads - 1) / kOrderThreads;
    k_group_order_count<<<blocks, kOrderThreads, 0, s>>>(len, groups, blockHist);
    k_group_order_scatter<<<blocks, kOrderThreads, 0, s>>>(len, groups, blockHist, order);
    return cudaGetLastError();
}

// Reference positionUpdater (tree.cu:678-703).
__global__ void __launch_bounds__(256)
k_kick_drift(float4* __restrict__ pos, float3* __restrict__ vel, const float3* __restrict__ acc, int n, float dt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float3 a = acc[i];
        float3 v = vel[i];
        float4 p = pos[i];
        v.x = __fmaf_rn(a.x, dt, v.x);
        v.y = __fmaf_rn(a.y, dt, v.y);
        v.z = __fmaf_rn(a.z, dt, v.z);
        p.x = __fmaf_rn(v.x, dt, p.x);
        p.y = __fmaf_rn(v.y, dt, p.y);
        p.z = __fmaf_rn(v.z, dt, p.z);
        vel[i] = v;
        pos[i] = p;
    }
}

// ---------------------------------------------------------------- launchers

int bh_walk_grid() { return bh_sm_count() * kBlocksPerSm; }
static_assert(kMinBlocksPlain <= kBlocksPerSm && kMinBlocksRelative <= kBlocksPerSm && kMinBlocksWide <= kBlocksPerSm &&
                  kMinBlocksFew <= kBlocksPerSm,
              "spill area sizing");

size_t bh_walk_spill_ints() { return (size_t)bh_walk_grid() * kWarpsPerBlock * kSpillPerWarp; }

// One walk variant: the persistent grid fills every SM with as many blocks as
// are resident at once for this stack size (registers or shared memory,
// whichever binds first, never more than the register budget the variant was
// compiled for).
template <typename Kernel>
static cudaError_t launch_walk_variant(Kernel kernel, const WalkArgs& a, int maxBlocks, bool wide, cudaStream_t s) {
    const size_t dyn = (size_t)kWarpsPerBlock * (wide ? WarpMem<true>::bytes(a.stackSmem) : WarpMem<false>::bytes(a.stackSmem));
    // deep stacks take the block past 48 KB of shared memory, which needs
    // the kernel's opt-in (a function attribute; harmless below that)
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    int resident = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kThreads, dyn);
    if (e != cudaSuccess) return e;
    resident = resident < maxBlocks ? resident : maxBlocks;
    if (resident < 1) return cudaErrorInvalidConfiguration;
    // How many warps share the groups.  A walk of few groups launches no warps
    // that would only find the cursor at its end, and its blocks spread over the
    // SMs (512 groups taken by the first warps of a full grid sat on few SMs: 155
    // us at 16,384 bodies, 93 with a grid of their own).  Where half of a
    // sub-partition's groups plus one is fewer than the warps that it could hold,
    // that many are walked at once: the groups come longest first, so a warp that
    // is done takes a short one, and fewer at once leave no half-empty last wave.
    // That is so at six to eight groups per sub-partition in the build for many
    // groups and at four in the 64-body one, both 113,665 to 151,552 bodies; below,
    // the few-groups build holds no more than three and takes them all.  Walk of
    // theta 0.5 disks / Plummer spheres, us, all warps and this many: 114,000 bodies
    // 239 / 241 and 211 / 215, 128,000 246 / 246 and 221 / 230, 144,000 250 / 254 and
    // 224 / 248; learned 306 / 458 and 298 / 469, 321 / 518 and 303 / 496, 334 / 524 and
    // 321 / 474; 64-body groups at 128,000 336 / 325 and 280 / 275.  Without an order
    // (accelerations of a state, the drop-in walk) build and walk together are the
    // same within 2%.
    const int perGroup = wide ? 64 : 32, sms = bh_sm_count();
    const long long groups = a.groupTable ? a.groups : (a.n + perGroup - 1) / perGroup;
    const long long half = (groups - 1) / (2ll * kWarpsPerBlock * sms) + 1;  // rounded up
    const int perSm = half + 1 < resident ? (int)half + 1 : resident;
    const long long all = (long long)sms * perSm, some = (groups + kWarpsPerBlock - 1) / kWarpsPerBlock;
    kernel<<<(unsigned)(some < all ? some : all), kThreads, dyn, s>>>(a);
    return cudaGetLastError();
}

int bh_walk_stack_default() { return kStackSmemDefault; }

cudaError_t bh_launch_walk(const WalkArgs& in, bool fused, bool compensated, cudaStream_t s) {
    WalkArgs a = in;
    if (a.stackSmem == 0) a.stackSmem = kStackSmemDefault;
    if (a.stackSmem < BH_WALK_STACK_MIN || a.stackSmem > BH_WALK_STACK_MAX || a.stackSmem % 32 != 0)
        return cudaErrorInvalidValue;
    if (a.relative && !a.aMagIn) return cudaErrorInvalidValue;
    const bool buckets = a.leafSize > 1;
    if (buckets && !a.nFirst) return cudaErrorInvalidValue;
    const int width = a.groupWidth ? a.groupWidth : 32;
    if (width != 32 && width != 64) return cudaErrorInvalidValue;
    const bool wide = width == 64;
    // one block per resident slot (the spill area is sized for bh_walk_grid(), the largest)
    const long long groups = a.groupTable ? a.groups : (a.n + 31) / 32;
    const bool few = !wide && groups <= (long long)kFewGroupsPerSm * bh_sm_count();
    const int maxBlocks = walk_min_blocks(a.relative, wide, few);
#define BH_WALK_LAUNCH(F, C, R, B, W, N) \
    return launch_walk_variant(k_walk<F, C, R, B, W, N>, a, maxBlocks, W, s)
#define BH_WALK_BUCKETS(F, C, R)                                      \
    do {                                                              \
        if (wide) {                                                   \
            if (buckets) BH_WALK_LAUNCH(F, C, R, true, true, false);  \
            else BH_WALK_LAUNCH(F, C, R, false, true, false);         \
        } else if (few) {                                             \
            if (buckets) BH_WALK_LAUNCH(F, C, R, true, false, true);  \
            else BH_WALK_LAUNCH(F, C, R, false, false, true);         \
        } else {                                                      \
            if (buckets) BH_WALK_LAUNCH(F, C, R, true, false, false); \
            else BH_WALK_LAUNCH(F, C, R, false, false, false);        \
        }                                                             \
    } while (0)
    if (a.relative) {
        if (fused) {
            if (compensated) BH_WALK_BUCKETS(true, true, true);
            else BH_WALK_BUCKETS(true, false, true);
        } else {
            if (compensated) BH_WALK_BUCKETS(false, true, true);
            else BH_WALK_BUCKETS(false, false, true);
        }
    } else {
        if (fused) {
            if (compensated) BH_WALK_BUCKETS(true, true, false);
            else BH_WALK_BUCKETS(true, false, false);
        } else {
            if (compensated) BH_WALK_BUCKETS(false, true, false);
            else BH_WALK_BUCKETS(false, false, false);
        }
    }
#undef BH_WALK_BUCKETS
#undef BH_WALK_LAUNCH
}

cudaError_t bh_launch_kick_drift(float4* pos, float3* vel, const float3* acc, int n, float dt,
                                 cudaStream_t s) {
    int grid = (n + 255) / 256;
    const int cap = 8 * bh_sm_count();
    grid = grid < 1 ? 1 : (grid > cap ? cap : grid);
    k_kick_drift<<<grid, 256, 0, s>>>(pos, vel, acc, n, dt);
    return cudaGetLastError();
}
