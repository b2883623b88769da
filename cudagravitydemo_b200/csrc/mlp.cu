// mlp.cu — the learned opening criterion: group features, a BF16 MLP
// (8 -> 32 -> 32 -> 1, ReLU, FP32 accumulation) on the tensor cores, its
// training (forward + backward + Adam) and the per-group choice of the
// relative-criterion budget.
//
// For a 32-body group and a candidate budget alpha, the MLP predicts
// log10 of the group's RMS relative force error under the relative opening
// criterion (walk.cu).  Per group, c = the largest candidate whose prediction
// meets the target; the budget is interpolated between candidates c and c+1
// where the predicted curve crosses the target (linear in log alpha), so a
// group's error sits at the target rather than up to a ladder step below it.
// A group whose predictions are not finite falls back to the reference's
// fixed-theta test (theta 0.5).
//
// Inputs (8): log10 alpha, then seven group features computed from the
// sorted bodies and the last step's accelerations (k_group_features).
// Matrix products use mma.sync m16n8k16 (BF16 in, FP32 accumulate): the
// network is 1.4k parameters, its GEMMs are 16 x 16 x 32 tiles, and a single
// warp-level MMA per tile is the right size for them.  The accumulator layout
// of one layer is the A-operand layout of the next, so layers chain in
// registers.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <math.h>

#include "bh_internal.cuh"
#include "bh_kernels.cuh"

namespace cg = cooperative_groups;

// ------------------------------------------------------------- parameters
// Packed FP32 parameter block (row-major W[in][out]):
//   W1[8][32] b1[32] W2[32][32] b2[32] W3[32] b3  + feature mean[8], scale[8]
#define MLP_W1 0
#define MLP_B1 256
#define MLP_W2 288
#define MLP_B2 1312
#define MLP_W3 1344
#define MLP_B3 1376
#define MLP_TRAINED 1377  // trained parameters
#define MLP_MU 1377
#define MLP_SIG 1385
#define MLP_TOTAL 1393

static_assert(MLP_TOTAL == BH_MLP_PARAMS, "parameter block size");
static_assert(MLP_TRAINED == BH_MLP_TRAINED, "trained parameter count");

// The budget ladder: alpha_c = kMacAlpha0 * 2^c, c = 0..BH_MAC_CANDIDATES-1
// (about 5e-4 to 1e-2 RMS relative force error on a disk galaxy).
constexpr float kMacAlpha0 = 2e-4f;
static_assert(BH_MAC_CANDIDATES == 8, "the selection kernel evaluates 8 candidates per group");

namespace {

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// D = A * B + C, m16n8k16, A/B bf16, C/D f32
__device__ __forceinline__ void mma_bf16(float d[4], const uint32_t a[4], const uint32_t b[2], const float c[4]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c[0]), "f"(c[1]), "f"(c[2]),
          "f"(c[3]));
}

// B fragment of a row-major weight W[in][out] (stride `out`) for the n-tile
// starting at column n0 and the k-step starting at row k0; rows >= kmax and
// columns >= nmax are zero.
__device__ __forceinline__ void load_b(uint32_t b[2], const float* W, int out, int k0, int n0, int kmax, int nmax) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n = n0 + g;
    auto w = [&](int k) { return (k < kmax && n < nmax) ? W[k * out + n] : 0.f; };
    b[0] = pack_bf16(w(k0 + 2 * t), w(k0 + 2 * t + 1));
    b[1] = pack_bf16(w(k0 + 2 * t + 8), w(k0 + 2 * t + 9));
}

// Warp-resident weights: B fragments of W1 (1 k-step x 4 n-tiles), W2 (2 x 4),
// W3 (2 x 1, 1 output) and the biases of this thread's columns.
struct MlpRegs {
    uint32_t w1[4][2], w2[2][4][2], w3[2][2];
    float b1[4][2], b2[4][2], b3;
    float mu[2], sig[2];  // normalisation of this thread's inputs 2t, 2t+1
};

__device__ void load_mlp(MlpRegs& r, const float* P) {
    const int t = threadIdx.x & 3;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        load_b(r.w1[j], P + MLP_W1, 32, 0, 8 * j, 8, 32);
        load_b(r.w2[0][j], P + MLP_W2, 32, 0, 8 * j, 32, 32);
        load_b(r.w2[1][j], P + MLP_W2, 32, 16, 8 * j, 32, 32);
        r.b1[j][0] = P[MLP_B1 + 8 * j + 2 * t];
        r.b1[j][1] = P[MLP_B1 + 8 * j + 2 * t + 1];
        r.b2[j][0] = P[MLP_B2 + 8 * j + 2 * t];
        r.b2[j][1] = P[MLP_B2 + 8 * j + 2 * t + 1];
    }
    load_b(r.w3[0], P + MLP_W3, 1, 0, 0, 32, 1);
    load_b(r.w3[1], P + MLP_W3, 1, 16, 0, 32, 1);
    r.b3 = P[MLP_B3];
#pragma unroll
    for (int f = 0; f < 2; f++) {
        r.mu[f] = P[MLP_MU + 2 * t + f];
        r.sig[f] = P[MLP_SIG + 2 * t + f];
    }
}

// Forward pass of a 16-row tile.  x0/x1: this thread's raw features 2t, 2t+1
// of rows g and g+8 (x0 = row g, x1 = row g+8).  Returns pre-activations z1,
// z2 (accumulator layout) and the output of rows g and g+8 (valid in threads
// with t == 0).
struct Acts {
    float z1[4][4], z2[4][4];
    float y[2];
};

__device__ void forward(const MlpRegs& r, const float x0[2], const float x1[2], Acts& a) {
    const int t = threadIdx.x & 3;
    uint32_t ax[4];
    ax[0] = pack_bf16((x0[0] - r.mu[0]) * r.sig[0], (x0[1] - r.mu[1]) * r.sig[1]);
    ax[1] = pack_bf16((x1[0] - r.mu[0]) * r.sig[0], (x1[1] - r.mu[1]) * r.sig[1]);
    ax[2] = ax[3] = 0u;  // features 8..15: padding
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float c[4] = {r.b1[j][0], r.b1[j][1], r.b1[j][0], r.b1[j][1]};
        mma_bf16(a.z1[j], ax, r.w1[j], c);
    }
    uint32_t ah[2][4];  // relu(z1) as the A operand of layer 2 (k-steps 0, 1)
#pragma unroll
    for (int s = 0; s < 2; s++) {
        ah[s][0] = pack_bf16(fmaxf(a.z1[2 * s][0], 0.f), fmaxf(a.z1[2 * s][1], 0.f));
        ah[s][1] = pack_bf16(fmaxf(a.z1[2 * s][2], 0.f), fmaxf(a.z1[2 * s][3], 0.f));
        ah[s][2] = pack_bf16(fmaxf(a.z1[2 * s + 1][0], 0.f), fmaxf(a.z1[2 * s + 1][1], 0.f));
        ah[s][3] = pack_bf16(fmaxf(a.z1[2 * s + 1][2], 0.f), fmaxf(a.z1[2 * s + 1][3], 0.f));
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float c[4] = {r.b2[j][0], r.b2[j][1], r.b2[j][0], r.b2[j][1]};
        mma_bf16(a.z2[j], ah[0], r.w2[0][j], c);
        mma_bf16(a.z2[j], ah[1], r.w2[1][j], a.z2[j]);
    }
    uint32_t ah2[2][4];
#pragma unroll
    for (int s = 0; s < 2; s++) {
        ah2[s][0] = pack_bf16(fmaxf(a.z2[2 * s][0], 0.f), fmaxf(a.z2[2 * s][1], 0.f));
        ah2[s][1] = pack_bf16(fmaxf(a.z2[2 * s][2], 0.f), fmaxf(a.z2[2 * s][3], 0.f));
        ah2[s][2] = pack_bf16(fmaxf(a.z2[2 * s + 1][0], 0.f), fmaxf(a.z2[2 * s + 1][1], 0.f));
        ah2[s][3] = pack_bf16(fmaxf(a.z2[2 * s + 1][2], 0.f), fmaxf(a.z2[2 * s + 1][3], 0.f));
    }
    float o[4] = {r.b3, 0.f, r.b3, 0.f};
    mma_bf16(o, ah2[0], r.w3[0], o);
    mma_bf16(o, ah2[1], r.w3[1], o);
    a.y[0] = o[0];  // row g, column 0 (threads with t == 0)
    a.y[1] = o[2];  // row g + 8
}

}  // namespace

// ---------------------------------------------------------------- features
// Seven features of each 32-body group (sorted order), from the bodies, the
// last step's |a| and the tree: see bh_group_features() in bh_api.h.
__global__ void __launch_bounds__(256)
k_group_features(const float4* __restrict__ pos, const float* __restrict__ aMag, const uint64_t* __restrict__ keys,
                 int n, int bits, const DevBox* __restrict__ box, const DevRoot* __restrict__ root, float G,
                 float* __restrict__ feat) {
    const int lane = threadIdx.x & 31;
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int groups = (n + 31) >> 5;
    if (g >= groups) return;
    const int b = g * 32 + lane;
    const bool valid = b < n;
    const float4 p = valid ? pos[b] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float am = valid ? aMag[b] : 0.f;
    float lo[3] = {valid ? p.x : INFINITY, valid ? p.y : INFINITY, valid ? p.z : INFINITY};
    float hi[3] = {valid ? p.x : -INFINITY, valid ? p.y : -INFINITY, valid ? p.z : -INFINITY};
    float aMin = valid ? am : INFINITY, aMax = valid ? am : 0.f, aSum = am, mSum = valid ? p.w : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
        aMin = fminf(aMin, __shfl_xor_sync(0xffffffffu, aMin, o));
        aMax = fmaxf(aMax, __shfl_xor_sync(0xffffffffu, aMax, o));
        aSum += __shfl_xor_sync(0xffffffffu, aSum, o);
        mSum += __shfl_xor_sync(0xffffffffu, mSum, o);
    }
    if (lane != 0) return;
    const int cnt = (n - g * 32 < 32) ? n - g * 32 : 32;
    const float ext = fmaxf(box->extent, 1e-30f);
    // the system's centre of mass and total mass from the FP64 root reduction
    const float mTot = (float)root->mass;
    const float hx = 0.5f * (hi[0] - lo[0]), hy = 0.5f * (hi[1] - lo[1]), hz = 0.5f * (hi[2] - lo[2]);
    const float R = sqrtf(hx * hx + hy * hy + hz * hz);
    const float cx = (float)((double)(0.5f * (lo[0] + hi[0])) - root->com[0]),
                cy = (float)((double)(0.5f * (lo[1] + hi[1])) - root->com[1]),
                cz = (float)((double)(0.5f * (lo[2] + hi[2])) - root->com[2]);
    const float D = sqrtf(cx * cx + cy * cy + cz * cz);
    const float aMean = aSum / cnt;
    const float aScale = G * fmaxf(mTot, 1e-30f) / (ext * ext);
    const uint64_t x = keys[g * 32] ^ keys[g * 32 + cnt - 1];
    const int depth = (x == 0ull) ? bits : bits - 1 - (63 - __clzll((long long)x)) / 3;
    const float vol = fmaxf(8.f * hx * hy * hz, 1e-30f * ext * ext * ext);
    const float hmin = fminf(hx, fminf(hy, hz)), hmax = fmaxf(hx, fmaxf(hy, hz));
    float* f = feat + (size_t)g * 7;
    f[0] = log10f(R / ext + 1e-7f);                                       // group radius
    f[1] = log10f(aMean / aScale + 1e-12f);                               // force scale
    f[2] = log10f((aMax + 1e-30f) / (aMin + 1e-30f));                     // force spread in the group
    f[3] = log10f(D / ext + 1e-4f);                                       // distance from the centre
    f[4] = (float)depth / (float)bits;                                    // tree depth of the group
    f[5] = log10f(mSum / fmaxf(mTot, 1e-30f) * ext * ext * ext / vol);   // local density
    f[6] = log10f((hmin + 1e-7f * ext) / (hmax + 1e-7f * ext));           // flatness
}

// --------------------------------------------------------------- inference
// Per group, evaluate the MLP at the kMacCandidates budgets and choose.
__global__ void __launch_bounds__(128)
k_mac_select(const float* __restrict__ P, const float* __restrict__ feat, int groups, float logTarget, float thetaCap,
             float2* __restrict__ groupParam) {
    MlpRegs r;
    load_mlp(r, P);
    const int lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    // a 16-row tile = 2 groups x 8 candidates: row = 8 * (group in tile) + candidate
    for (int tile = warp; tile * 2 < groups; tile += nwarps) {
        const int gA = tile * 2, gB = gA + 1;
        // row g8 -> group gA, candidate g8; row g8 + 8 -> group gB, candidate g8
        float x0[2], x1[2];
        auto feature = [&](int grp, int cand, int f) -> float {
            if (grp >= groups) return 0.f;
            return f == 0 ? log10f(ldexpf(kMacAlpha0, cand)) : feat[(size_t)grp * 7 + f - 1];
        };
        x0[0] = feature(gA, g8, 2 * t);
        x0[1] = feature(gA, g8, 2 * t + 1);
        x1[0] = feature(gB, g8, 2 * t);
        x1[1] = feature(gB, g8, 2 * t + 1);
        Acts a;
        forward(r, x0, x1, a);
        // lanes with t == 0 hold rows g8 (group A) and g8 + 8 (group B)
        const float yA = __shfl_sync(0xffffffffu, a.y[0], (lane & ~3));
        const float yB = __shfl_sync(0xffffffffu, a.y[1], (lane & ~3));
        // lane (4c + t), t == 0 carries candidate c: ballots over candidates
        const bool finiteA = isfinite(yA), finiteB = isfinite(yB);
        const unsigned okA = __ballot_sync(0xffffffffu, t == 0 && finiteA && yA <= logTarget);
        const unsigned okB = __ballot_sync(0xffffffffu, t == 0 && finiteB && yB <= logTarget);
        const unsigned badA = __ballot_sync(0xffffffffu, t == 0 && !finiteA);
        const unsigned badB = __ballot_sync(0xffffffffu, t == 0 && !finiteB);
        // largest budget that meets the target (uniform), its prediction and the next one's
        const int cA = okA ? (31 - __clz(okA)) >> 2 : 0, cB = okB ? (31 - __clz(okB)) >> 2 : 0;
        const float ycA = __shfl_sync(0xffffffffu, yA, 4 * cA), ycB = __shfl_sync(0xffffffffu, yB, 4 * cB);
        const float ynA = __shfl_sync(0xffffffffu, yA, cA < 7 ? 4 * cA + 4 : 28);
        const float ynB = __shfl_sync(0xffffffffu, yB, cB < 7 ? 4 * cB + 4 : 28);
        if (lane == 0) {
            auto pick = [&](unsigned ok, unsigned bad, int c, float yc, float yn) -> float2 {
                if (bad) return make_float2(0.5f, 1e30f);  // fallback: the fixed-theta test alone
                float alpha = ldexpf(kMacAlpha0, c);
                // c meets the target and c+1 does not: interpolate in log alpha
                if (ok && c < BH_MAC_CANDIDATES - 1 && yn > logTarget && yn > yc) {
                    const float frac = __fdiv_rn(__fsub_rn(logTarget, yc), __fsub_rn(yn, yc));
                    alpha = __fmul_rn(alpha, exp2f(frac));
                }
                return make_float2(thetaCap, alpha);
            };
            groupParam[gA] = pick(okA, badA, cA, ycA, ynA);
            if (gB < groups) groupParam[gB] = pick(okB, badB, cB, ycB, ynB);
        }
    }
}

// ---------------------------------------------------------------- training
// A warp takes 16 rows: forward and the backward product through W2 on the
// tensor cores (BF16 in, FP32 out), then the weight gradients as FP32 sums over
// the rows, each lane one column of every matrix in registers, which 16 rows of
// activations pass by in shared memory (a column's values are loaded lane by
// lane, what they are multiplied with comes as broadcasts).  The sums of a
// block's warps meet in shared memory at the end of a batch.
namespace {
// floats a row keeps: x 0..7, then h1, dh2, dh1, h2 (32 each); 8 more than a
// multiple of 32, so that four rows' pairs are stored without bank conflicts
constexpr int kRow = 136, kH1 = 8, kD2 = 40, kD1 = 72, kH2 = 104;
constexpr int kDy = 16 * kRow;           // after a warp's 16 rows: dy of each
constexpr int kWarpRows = kDy + 16;      // floats of a warp
constexpr int kRed = 1408;               // MLP_TRAINED rounded up

// Gradient sums of one lane: W2[i][lane], W1[f][lane], b1[lane], b2[lane],
// W3[lane], and its share of b3.
struct Grads {
    float w2[32], w1[8], b1, b2, w3, b3;
};

__device__ __forceinline__ void clear(Grads& q) {
#pragma unroll
    for (int i = 0; i < 32; i++) q.w2[i] = 0.f;
#pragma unroll
    for (int f = 0; f < 8; f++) q.w1[f] = 0.f;
    q.b1 = q.b2 = q.w3 = q.b3 = 0.f;
}

// One lane's inputs of a 16-row tile: features 2t, 2t+1 of rows g and g + 8,
// and their targets; rows past the end are zero and marked.
struct TileIn {
    float2 x0, x1;
    float y0, y1;
    bool has0, has1;
};

__device__ __forceinline__ TileIn load_tile(const float* __restrict__ X, const float* __restrict__ Y, int r0, int rows) {
    const int lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
    TileIn in;
    const int ra = r0 + g8, rb = ra + 8;
    in.has0 = ra < rows;
    in.has1 = rb < rows;
    in.x0 = in.x1 = make_float2(0.f, 0.f);
    in.y0 = in.y1 = 0.f;
    if (in.has0) {
        in.x0 = make_float2(X[(size_t)ra * 8 + 2 * t], X[(size_t)ra * 8 + 2 * t + 1]);
        in.y0 = Y[ra];
    }
    if (in.has1) {
        in.x1 = make_float2(X[(size_t)rb * 8 + 2 * t], X[(size_t)rb * 8 + 2 * t + 1]);
        in.y1 = Y[rb];
    }
    return in;
}

// Adds one tile's gradients of sum (MLP(x) - y)^2 / rows to q and its squared
// errors to loss.  P: parameters and the fragments made of them, in shared
// memory (frag[k][lane], k as in make_fragments); S: this warp's 16 rows.
constexpr int kFrag = 44;  // W1: 0..7, W2: 8..23, W3: 24..27, W2 transposed: 28..43
__device__ void tile_gradients(const float* P, const uint32_t* frag, const TileIn& in, float dyScale, float* S, Grads& q,
                               float& loss) {
    const int lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
    const uint32_t* F = frag + lane;
    auto fragment = [&](uint32_t b[2], int k) {
        b[0] = F[32 * k];
        b[1] = F[32 * (k + 1)];
    };
    float* const S0 = S + g8 * kRow;
    float* const S1 = S0 + 8 * kRow;
    auto put = [](float* at, float a, float b) { *reinterpret_cast<float2*>(at) = make_float2(a, b); };
    // two values as a product sees them, rounded to bf16
    auto putRounded = [&](float* at, uint32_t two) { put(at, __uint_as_float(two << 16), __uint_as_float(two & 0xffff0000u)); };
    uint32_t ax[4];
    {
        const float2 mu = make_float2(P[MLP_MU + 2 * t], P[MLP_MU + 2 * t + 1]);
        const float2 sig = make_float2(P[MLP_SIG + 2 * t], P[MLP_SIG + 2 * t + 1]);
        const float a0 = (in.x0.x - mu.x) * sig.x, a1 = (in.x0.y - mu.y) * sig.y;
        const float b0 = (in.x1.x - mu.x) * sig.x, b1 = (in.x1.y - mu.y) * sig.y;
        ax[0] = pack_bf16(a0, a1);
        ax[1] = pack_bf16(b0, b1);
        ax[2] = ax[3] = 0u;  // features 8..15: padding
        // normalised, bf16-rounded inputs (what the products saw)
        putRounded(S0 + 2 * t, ax[0]);
        putRounded(S1 + 2 * t, ax[1]);
    }
    float z1[4][4], z2[4][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 b = make_float2(P[MLP_B1 + 8 * j + 2 * t], P[MLP_B1 + 8 * j + 2 * t + 1]);
        const float c[4] = {b.x, b.y, b.x, b.y};
        uint32_t w[2];
        fragment(w, 2 * j);
        mma_bf16(z1[j], ax, w, c);
    }
    uint32_t ah[2][4];  // relu(z1) as the A operand of layer 2 (k-steps 0, 1)
    auto activate = [&](const float z[4][4], int col) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float h0 = fmaxf(z[j][0], 0.f), h1 = fmaxf(z[j][1], 0.f), h2 = fmaxf(z[j][2], 0.f), h3 = fmaxf(z[j][3], 0.f);
            ah[j >> 1][2 * (j & 1)] = pack_bf16(h0, h1);
            ah[j >> 1][2 * (j & 1) + 1] = pack_bf16(h2, h3);
            putRounded(S0 + col + 8 * j + 2 * t, ah[j >> 1][2 * (j & 1)]);
            putRounded(S1 + col + 8 * j + 2 * t, ah[j >> 1][2 * (j & 1) + 1]);
        }
    };
    activate(z1, kH1);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float2 b = make_float2(P[MLP_B2 + 8 * j + 2 * t], P[MLP_B2 + 8 * j + 2 * t + 1]);
        const float c[4] = {b.x, b.y, b.x, b.y};
        uint32_t w[2];
        fragment(w, 8 + 2 * j);
        mma_bf16(z2[j], ah[0], w, c);
        fragment(w, 16 + 2 * j);
        mma_bf16(z2[j], ah[1], w, z2[j]);
    }
    activate(z2, kH2);
    float o[4] = {P[MLP_B3], 0.f, P[MLP_B3], 0.f};
    {
        uint32_t w[2];
        fragment(w, 24);
        mma_bf16(o, ah[0], w, o);
        fragment(w, 26);
        mma_bf16(o, ah[1], w, o);
    }
    // dL/dy = 2 (y - target) / rows, from the lanes of column 0 (rows past the
    // end contribute nothing)
    float dy0 = 0.f, dy1 = 0.f;
    if (t == 0) {
        const float da = in.has0 ? o[0] - in.y0 : 0.f, db = in.has1 ? o[2] - in.y1 : 0.f;
        loss += da * da + db * db;
        dy0 = 2.f * da / dyScale;
        dy1 = 2.f * db / dyScale;
        S[kDy + g8] = dy0;
        S[kDy + g8 + 8] = dy1;
    }
    dy0 = __shfl_sync(0xffffffffu, dy0, lane & ~3);
    dy1 = __shfl_sync(0xffffffffu, dy1, lane & ~3);
    // dh2 = dy * W3 * relu'(z2), and as the A operand (bf16) of dh1 = dh2 W2^T
    uint32_t ad[2][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = 8 * j + 2 * t;
        const float w0 = bf16_round(P[MLP_W3 + c]), w1 = bf16_round(P[MLP_W3 + c + 1]);
        const float d0 = z2[j][0] > 0.f ? dy0 * w0 : 0.f, d1 = z2[j][1] > 0.f ? dy0 * w1 : 0.f;
        const float d2 = z2[j][2] > 0.f ? dy1 * w0 : 0.f, d3 = z2[j][3] > 0.f ? dy1 * w1 : 0.f;
        ad[j >> 1][2 * (j & 1)] = pack_bf16(d0, d1);
        ad[j >> 1][2 * (j & 1) + 1] = pack_bf16(d2, d3);
        put(S0 + kD2 + c, d0, d1);
        put(S1 + kD2 + c, d2, d3);
    }
    // dh1[r][i] = sum_j dh2[r][j] W2[i][j] * relu'(z1[r][i])
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t w[2];
        fragment(w, 28 + 4 * j);
        mma_bf16(acc, ad[0], w, acc);
        fragment(w, 28 + 4 * j + 2);
        mma_bf16(acc, ad[1], w, acc);
        const int c = 8 * j + 2 * t;
        put(S0 + kD1 + c, z1[j][0] > 0.f ? acc[0] : 0.f, z1[j][1] > 0.f ? acc[1] : 0.f);
        put(S1 + kD1 + c, z1[j][2] > 0.f ? acc[2] : 0.f, z1[j][3] > 0.f ? acc[3] : 0.f);
    }
    __syncwarp();
    const float* R = S;
#pragma unroll 2
    for (int r = 0; r < 16; r++, R += kRow) {
        const float d1 = R[kD1 + lane], d2 = R[kD2 + lane];
#pragma unroll
        for (int f = 0; f < 8; f += 4) {
            const float4 x = *reinterpret_cast<const float4*>(R + f);
            q.w1[f] = fmaf(x.x, d1, q.w1[f]);
            q.w1[f + 1] = fmaf(x.y, d1, q.w1[f + 1]);
            q.w1[f + 2] = fmaf(x.z, d1, q.w1[f + 2]);
            q.w1[f + 3] = fmaf(x.w, d1, q.w1[f + 3]);
        }
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            const float4 h = *reinterpret_cast<const float4*>(R + kH1 + i);
            q.w2[i] = fmaf(h.x, d2, q.w2[i]);
            q.w2[i + 1] = fmaf(h.y, d2, q.w2[i + 1]);
            q.w2[i + 2] = fmaf(h.z, d2, q.w2[i + 2]);
            q.w2[i + 3] = fmaf(h.w, d2, q.w2[i + 3]);
        }
        q.b1 += d1;
        q.b2 += d2;
        q.w3 = fmaf(R[kH2 + lane], S[kDy + r], q.w3);
    }
    if (lane < 16) q.b3 += S[kDy + lane];
    __syncwarp();
}

// The bf16 operand fragments of the weights, one word per lane each: W1 (4
// n-tiles), W2 (2 k-steps x 4 n-tiles), W3 (2 k-steps), W2 transposed (4 x 2).
__device__ void make_fragments(const float* P, uint32_t* frag, int threads) {
    for (int e = threadIdx.x; e < kFrag * 32; e += threads) {
        const int k = e >> 5, lane = e & 31, g = lane >> 2, t = lane & 3;
        const int half = (k & 1) * 8 + 2 * t;  // k index of the word's first value within a 16-deep k-step
        float a = 0.f, b = 0.f;
        if (k < 8) {  // W1[in][8 j + g], in < 8: the second word is padding
            const float* w = P + MLP_W1 + 8 * (k >> 1) + g;
            if (half < 8) { a = w[32 * half]; b = w[32 * (half + 1)]; }
        } else if (k < 24) {  // W2[16 s + half][8 j + g]
            const float* w = P + MLP_W2 + 32 * (16 * ((k - 8) >> 3) + half) + 8 * (((k - 8) >> 1) & 3) + g;
            a = w[0]; b = w[32];
        } else if (k < 28) {  // W3[16 s + half], one output
            const float* w = P + MLP_W3 + 16 * ((k - 24) >> 1) + half;
            if (g == 0) { a = w[0]; b = w[1]; }
        } else {  // W2[8 j + g][16 s + half]
            const float* w = P + MLP_W2 + 32 * (8 * ((k - 28) >> 2) + g) + 16 * (((k - 28) >> 1) & 1) + half;
            a = w[0]; b = w[1];
        }
        frag[e] = pack_bf16(a, b);
    }
}

// A warp's gradient sums into its row of red[warp][kRed].
__device__ void store_gradients(const Grads& q, float* red) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 32; i++) red[MLP_W2 + i * 32 + lane] = q.w2[i];
#pragma unroll
    for (int f = 0; f < 8; f++) red[MLP_W1 + f * 32 + lane] = q.w1[f];
    red[MLP_B1 + lane] = q.b1;
    red[MLP_B2 + lane] = q.b2;
    red[MLP_W3 + lane] = q.w3;
    float b3 = q.b3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b3 += __shfl_xor_sync(0xffffffffu, b3, o);
    if (lane == 0) red[MLP_B3] = b3;
}

// Shared memory of a block of `warps` warps: parameters, fragments, and the
// rows, whose place the warps' sums take at the end of a batch.
constexpr int kParams = 1396;  // MLP_TOTAL rounded up to 16 bytes
constexpr size_t train_smem(int warps) {
    const size_t rows = (size_t)warps * kWarpRows, sums = (size_t)warps * kRed;
    return 4 * (kParams + kFrag * 32 + (rows > sums ? rows : sums));
}
constexpr int kGradWarps = 4, kEpochWarps = 16, kMaxCluster = 16;

// One Adam step of one parameter (its roundings spelled out, so that both
// kernels that take it agree): moments updated, the new parameter returned.
__device__ __forceinline__ float adam_step(float p, float g, float& m, float& v, float lr, float b1, float b2, float eps,
                                           float c1, float c2) {
    m = __fmaf_rn(1.f - b1, g, __fmul_rn(b1, m));
    v = __fmaf_rn(__fmul_rn(1.f - b2, g), g, __fmul_rn(b2, v));
    return __fsub_rn(p, __fdiv_rn(__fmul_rn(lr, __fdiv_rn(m, c1)), __fadd_rn(__fsqrt_rn(__fdiv_rn(v, c2)), eps)));
}

// Sum of 16 in a tree: four roundings on each value's way instead of fifteen.
__device__ __forceinline__ float pairwise_sum(float (&v)[16]) {
#pragma unroll
    for (int half = 8; half > 0; half >>= 1)
#pragma unroll
        for (int k = 0; k < half; k++) v[k] += v[k + half];
    return v[0];
}
}  // namespace

// Gradient and loss over `rows` rows, any grid: the blocks' sums meet in grad
// and lossOut by atomics (both zeroed by the caller).
__global__ void __launch_bounds__(kGradWarps * 32)
k_mlp_grad(const float* __restrict__ P, const float* __restrict__ X, const float* __restrict__ Y, int rows,
           float* __restrict__ grad, float* __restrict__ lossOut) {
    extern __shared__ __align__(16) float sh[];
    float* const sP = sh;
    uint32_t* const frag = reinterpret_cast<uint32_t*>(sP + kParams);
    float* const rowsMem = sP + kParams + kFrag * 32;
    for (int i = threadIdx.x; i < MLP_TOTAL; i += blockDim.x) sP[i] = P[i];
    __syncthreads();
    make_fragments(sP, frag, kGradWarps * 32);
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Grads q;
    clear(q);
    float loss = 0.f;
    for (int tile = blockIdx.x * kGradWarps + w; tile * 16 < rows; tile += gridDim.x * kGradWarps)
        tile_gradients(sP, frag, load_tile(X, Y, tile * 16, rows), (float)rows, rowsMem + w * kWarpRows, q, loss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) atomicAdd(lossOut, loss);
    __syncthreads();
    store_gradients(q, rowsMem + w * kRed);
    __syncthreads();
    for (int i = threadIdx.x; i < MLP_TRAINED; i += blockDim.x) {
        float s = rowsMem[i];
#pragma unroll
        for (int k = 1; k < kGradWarps; k++) s += rowsMem[k * kRed + i];
        if (s != 0.f) atomicAdd(&grad[i], s);
    }
}

// A whole epoch in one launch of one cluster: every batch needs the parameters
// that the batch before it left, so a batch is a chain, and the chain is what
// bounds an epoch (23 us a batch as three launches of memset, gradient and Adam).
// Here the blocks share a batch's tiles, each sums its gradients, block r reads
// slice r of all blocks' sums over distributed shared memory (in block order),
// applies Adam to it in registers (FP32 master weights) and hands the new slice
// to every block; two cluster barriers a batch, no global memory but the rows.
// 1M rows in batches of 4,096: 5.87 -> 2.31 ms, 262,144 in batches of 500: 11.9
// -> 2.9 ms.  42% of a batch is instruction issue on the 16 SMs (two thirds of
// it the FP32 gradient sums), the rest the chain of barriers and latencies.
__global__ void __launch_bounds__(kEpochWarps * 32, 1)
k_mlp_epoch(float* __restrict__ P, const float* __restrict__ X, const float* __restrict__ Y, int rows, int batch,
            float* __restrict__ grad, float* __restrict__ adamM, float* __restrict__ adamV, double pow1, double pow2,
            float lr, float* __restrict__ lossOut) {
    constexpr int kThr = kEpochWarps * 32;
    constexpr float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    extern __shared__ __align__(16) float sh[];
    float* const sP = sh;
    uint32_t* const frag = reinterpret_cast<uint32_t*>(sP + kParams);
    float* const sum = sP + kParams + kFrag * 32;
    float* const rowsMem = sum + kRed;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), size = (int)cluster.num_blocks();
    const int slice = (MLP_TRAINED + size - 1) / size;
    const int own = rank * slice + (int)threadIdx.x;  // the parameter this thread steps, if any
    const bool mine = (int)threadIdx.x < slice && own < MLP_TRAINED;
    float m = mine ? adamM[own] : 0.f, v = mine ? adamV[own] : 0.f, g = 0.f;
    for (int i = threadIdx.x; i < MLP_TOTAL; i += kThr) sP[i] = P[i];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int tile0 = w * size + rank, tiles = kEpochWarps * size;  // a short batch spreads over the blocks
    float loss = 0.f;
    TileIn in = load_tile(X, Y, tile0 * 16, batch < rows ? batch : rows);
    for (int r0 = 0;; r0 += batch) {
        const int nb = rows - r0 < batch ? rows - r0 : batch;
        const bool more = nb < rows - r0;
        __syncthreads();  // the parameters are there
        make_fragments(sP, frag, kThr);
        __syncthreads();
        Grads q;
        clear(q);
        for (int tile = tile0; tile * 16 < nb; tile += tiles) {
            const TileIn now = in;
            if ((tile + tiles) * 16 < nb) in = load_tile(X + (size_t)r0 * 8, Y + r0, (tile + tiles) * 16, nb);
            tile_gradients(sP, frag, now, (float)nb, rowsMem + w * kWarpRows, q, loss);
        }
        // the next batch's rows come while this one's sums travel
        if (more) {
            const int next = rows - r0 - nb < batch ? rows - r0 - nb : batch;
            in = load_tile(X + (size_t)(r0 + nb) * 8, Y + r0 + nb, tile0 * 16, next);
        }
        __syncthreads();
        store_gradients(q, rowsMem + w * kRed);
        __syncthreads();
        for (int i = threadIdx.x; i < MLP_TRAINED; i += kThr) {
            float part[kEpochWarps];
#pragma unroll
            for (int k = 0; k < kEpochWarps; k++) part[k] = rowsMem[k * kRed + i];
            sum[i] = pairwise_sum(part);
        }
        cluster.sync();
        pow1 *= (double)b1;
        pow2 *= (double)b2;
        if (mine) {
            float part[kMaxCluster];  // all in flight at once; past the cluster's size zeros
#pragma unroll
            for (int k = 0; k < kMaxCluster; k++) part[k] = k < size ? cluster.map_shared_rank(sum, k)[own] : 0.f;
            g = pairwise_sum(part);
            const float c1 = 1.f - (float)pow1, c2 = 1.f - (float)pow2;
            const float p = adam_step(sP[own], g, m, v, lr, b1, b2, eps, c1, c2);
            for (int k = 0; k < size; k++) cluster.map_shared_rank(sP, k)[own] = p;
        }
        cluster.sync();
        if (!more) break;
    }
    if (mine) {
        P[own] = sP[own];
        adamM[own] = m;
        adamV[own] = v;
        grad[own] = g;  // the last batch's
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) atomicAdd(lossOut, loss);
}

// Adam on the trained parameters (FP32 master weights), for batches that have a
// launch of their own.
__global__ void k_adam(float* P, const float* grad, float* m, float* v, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= MLP_TRAINED) return;
    float mi = m[i], vi = v[i];
    P[i] = adam_step(P[i], grad[i], mi, vi, lr, b1, b2, eps, c1, c2);
    m[i] = mi;
    v[i] = vi;
}

namespace {
// grad += gradient, *loss += squared errors of `rows` rows, over the whole GPU
cudaError_t launch_grad(const float* params, const float* X, const float* Y, int rows, float* grad, float* loss,
                        cudaStream_t s) {
    constexpr size_t smem = train_smem(kGradWarps);
    static_assert(smem <= 48 * 1024, "k_mlp_grad needs no shared-memory opt-in");
    const int tiles = (rows - 1) / 16 + 1;
    int blocks = (tiles + kGradWarps - 1) / kGradWarps;
    blocks = blocks > 4 * bh_sm_count() ? 4 * bh_sm_count() : blocks;
    k_mlp_grad<<<blocks, kGradWarps * 32, smem, s>>>(params, X, Y, rows, grad, loss);
    return cudaGetLastError();
}

// Batches up to this many rows (two tiles per warp of the cluster) take the
// one-launch epoch; larger ones are better off on all SMs with two launches each
// (16,384 rows a batch, 1M rows: 1.64 ms in the cluster, 1.11 ms by launches; a
// single batch of 1M rows 1.35 and 0.20 ms).
constexpr int kEpochBatchMax = 8192;
}  // namespace

// ------------------------------------------------------------------ C ABI
extern "C" int bh_mlp_train_epoch(float* params, const float* X, const float* Y, int rows, float* grad, float* adamM,
                                  float* adamV, int batch, int* step, float lr, float* lossOut, cudaStream_t s) {
    if (!params || !X || !Y || rows <= 0 || !grad || !adamM || !adamV || batch <= 0 || !step || !lossOut)
        return BH_ERR_INVALID;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    if (batch > kEpochBatchMax && rows > kEpochBatchMax) {
        for (int r0 = 0;; r0 += batch) {
            const int nb = rows - r0 < batch ? rows - r0 : batch;
            BH_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(float) * MLP_TRAINED, s));
            BH_CUDA_TRY(launch_grad(params, X + (size_t)r0 * 8, Y + r0, nb, grad, lossOut, s));
            const int t = ++(*step);
            const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
            k_adam<<<(MLP_TRAINED + 255) / 256, 256, 0, s>>>(params, grad, adamM, adamV, lr, b1, b2, eps, c1, c2);
            BH_CUDA_TRY(cudaGetLastError());
            if (nb == rows - r0) return BH_OK;
        }
    }
    constexpr size_t smem = train_smem(kEpochWarps) + 4 * kRed;  // and the block's sums
    BH_CUDA_TRY(cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    BH_CUDA_TRY(cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kEpochWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // 16 blocks where the GPU can place such a cluster, else the portable 8
    for (int size = kMaxCluster;; size = 8) {
        cfg.gridDim = dim3(size);
        attr[0].val.clusterDim.x = size;
        int fit = 0;
        if (size == 8 || (cudaOccupancyMaxActiveClusters(&fit, k_mlp_epoch, &cfg) == cudaSuccess && fit > 0)) break;
    }
    (void)cudaGetLastError();
    const int before = *step, batches = (rows - 1) / batch + 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_mlp_epoch, params, X, Y, rows, batch, grad, adamM, adamV,
                                             pow((double)b1, before), pow((double)b2, before), lr, lossOut);
    if (e != cudaSuccess) return bh_note_cuda_error(e);
    *step = before + batches;
    return BH_OK;
}

extern "C" int bh_mlp_loss_grad(const float* params, const float* X, const float* Y, int rows, float* grad,
                                float* lossOut, cudaStream_t s) {
    if (!params || !X || !Y || rows <= 0 || !grad || !lossOut) return BH_ERR_INVALID;
    BH_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(float) * MLP_TRAINED, s));
    BH_CUDA_TRY(cudaMemsetAsync(lossOut, 0, sizeof(float), s));
    BH_CUDA_TRY(launch_grad(params, X, Y, rows, grad, lossOut, s));
    return BH_OK;
}

// Raw forward pass: Y[r] = MLP(X[r]) for `rows` rows of 8 inputs (a test and
// tooling entry; the selection kernel uses the same forward()).
__global__ void __launch_bounds__(128) k_mlp_forward(const float* P, const float* X, int rows, float* Y) {
    MlpRegs r;
    load_mlp(r, P);
    const int lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int tile = warp; tile * 16 < rows; tile += nwarps) {
        const int r0 = tile * 16;
        auto in = [&](int row, int f) { return row < rows ? X[(size_t)row * 8 + f] : 0.f; };
        const float x0[2] = {in(r0 + g8, 2 * t), in(r0 + g8, 2 * t + 1)};
        const float x1[2] = {in(r0 + g8 + 8, 2 * t), in(r0 + g8 + 8, 2 * t + 1)};
        Acts a;
        forward(r, x0, x1, a);
        if (t == 0) {
            if (r0 + g8 < rows) Y[r0 + g8] = a.y[0];
            if (r0 + g8 + 8 < rows) Y[r0 + g8 + 8] = a.y[1];
        }
    }
}

extern "C" int bh_mlp_forward(const float* params, const float* X, int rows, float* Y, cudaStream_t s) {
    if (!params || !X || !Y || rows <= 0) return BH_ERR_INVALID;
    const int tiles = (rows + 15) / 16;
    int blocks = (tiles + 3) / 4;
    blocks = blocks > 4 * bh_sm_count() ? 4 * bh_sm_count() : blocks;
    k_mlp_forward<<<blocks, 128, 0, s>>>(params, X, rows, Y);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? BH_OK : bh_note_cuda_error(e);
}

// ---------------------------------------------------------- engine hooks
cudaError_t bh_launch_group_features(const float4* pos, const float* aMag, const uint64_t* keys, int n, int bits,
                                     const DevBox* box, const DevRoot* root, float G, float* feat, cudaStream_t s) {
    const int groups = (n + 31) / 32;
    k_group_features<<<(groups + 7) / 8, 256, 0, s>>>(pos, aMag, keys, n, bits, box, root, G, feat);
    return cudaGetLastError();
}

cudaError_t bh_launch_mac_select(const float* params, const float* feat, int groups, float logTarget, float thetaCap,
                                 float2* groupParam, cudaStream_t s) {
    const int tiles = (groups + 1) / 2;
    int blocks = (tiles + 3) / 4;
    blocks = blocks > 8 * bh_sm_count() ? 8 * bh_sm_count() : blocks;
    blocks = blocks < 1 ? 1 : blocks;
    k_mac_select<<<blocks, 128, 0, s>>>(params, feat, groups, logTarget, thetaCap, groupParam);
    return cudaGetLastError();
}

extern "C" int bh_mac_ladder(float alphas[BH_MAC_CANDIDATES]) {
    if (!alphas) return BH_ERR_INVALID;
    for (int c = 0; c < BH_MAC_CANDIDATES; c++) alphas[c] = ldexpf(kMacAlpha0, c);
    return BH_OK;
}
