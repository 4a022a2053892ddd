// prefill_exact.cu -- causal attention of several query rows in f32 arithmetic, over the f32 or fp16 store, without
// scratch: what a session without room for fp16 twins runs, and the launches whose position lives on the device.
//
// What it replaces: kWarpAttention / kWarpAttentionPos and kQ35WarpAttention of the reference
// (include/gpu/GpuAttentionKernels.hpp:211-272, 537-599; include/gpu/GpuQwen35Kernels.hpp:2437-2492): row s attends
// cache rows [0, pos + s], score = dot(q, k) * invSqrt, online softmax with exp2, out = sum p v / sum p.
//
// Over the f32 store every operand is an fp16 pair, x = 2^e (hi + 2^-11 lo) with a power of two for the rows that a warp takes apart at a
// time (16, 8, 2 at head_dim 64, 128, 256), and a product is three on the
// tensor cores (mma.sync.m16n8k16: hi*hi + lo*hi + hi*lo, f32 accumulation): 22 bits of every factor like 3xTF32, at half the
// products and half the shared memory.  K's power goes into the score, V's into the probability, which has one of its own per query row.
// The pairs hold 22 bits over 2^29; f32 has no such limit.  So the warps that make them look for numbers outside it, and where those can count --
// outliers of 10^8 in a dim, rows of 2^40 next to others, infinities -- the blocks concerned go on in f32 (the second
// loop of the kernel): right, and some seven times slower (512 rows of 14 / 2 / 64 13.7 -> 78 - 87 us).
//
// What bounds it: shared memory and mma.sync in turn, and the loaders' instructions.  With 8 query rows at a time (the causal form of the decode
// kernels, which stays for few rows behind a long prefix: prefillExactWins below) every warp takes K and V apart for itself.  Here a block
// of 32 query rows of one q head does that once per stage, into planes in shared memory: loader warps (loads, exponents, the pairs)
// fill one buffer while the computing warps, 16 rows x TG tokens each, work on the other.  Done by the
// computing warps between two barriers, as tf32 planes, a stage of 128 tokens at head_dim 64 took 3.9 us (1.6 of them products);
// like this 2.3.  The
// four token groups of a block take their share of every stage (a short prompt is a chain of stages, not a matter of
// bytes) and are put together at the end.  The late rows of all heads come first, so that what starts last is short.
// Measured, tf32 planes -> this: 512 rows of 14 / 2 / 64 17.7 -> 13.7 us, 512 behind 3000 200 -> 122; 512 rows of 28 / 4 / 128
// 59 -> 43, 512 behind 512 178 -> 123; 512 rows of 16 / 2 / 256 75 -> 44, 512 behind 512 215 -> 114.  fp16 store, 8-row form -> this: 100
// rows of 28 / 4 / 128 15.0 -> 6.4 us, 512 behind 512 107 -> 71, 2000 rows of 8 / 4 / 64 81 -> 40.  (The look at the range and the powers per
// query row cost 6 - 10 % at head_dim 64 and 3 - 6 at 128; a power per row of K and V instead of one per unit as much again.)
//
// What keeps it exact: a tensor-core product drops the bits of a running sum that do not fit, and those losses add up
// along a chain.  So a stage's products are summed by themselves, the small terms apart (f32) or first (fp16), and added to O in
// f32.  Against a 64-bit evaluation, tf32 planes -> this: 512 rows behind 3000 of 14 / 2 / 64 4.0e-7 -> 3.0e-7 of the result's norm, of
// 8 / 2 / 128 (whose stages shared one sum) 5.9e-6 -> 3.6e-7; 512 behind 512 of 16 / 2 / 256 2.0e-6 -> 5.4e-7; fp16 512 behind 1000 2.9e-7.
#include "decode_cluster.cuh"

namespace tc {

struct PrefillExactParams {
    const float *q;
    float *out;
    const void *k, *v;        // [totalRows][nKV][HD]
    const uint32_t *devPos;   // nullable: position of row 0, read at kernel time
    uint64_t totalRows;
    uint32_t qRows, cachePos, nHeads, nKV, group;
    float scaleLog2;          // invSqrt * log2(e)
};

// RT 16-row tiles of query rows x NH token groups = warps that compute.
static constexpr int kExactRT = 2, kExactNH = 4, kExactWarps = kExactRT * kExactNH, kExactRows = 16 * kExactRT;
static constexpr uint32_t kExactThreads = kExactWarps * 32, kFoldBar = 1;  // (named barrier of those warps)

// TG tokens of a stage per group; NB stages of K and of V in shared memory.
template <int HD>
struct ExactShape {
    static constexpr int TG = HD == 64 ? 32 : 16, kRows = kExactRows, kStage = kExactNH * TG, NB = HD > 128 ? 1 : 2;
    static constexpr int kLoaders = 8, kThreads = (kExactWarps + kLoaders) * 32;
    // registers of a thread, and of a loader's: together what the launch has (512 x 128, 384 x 168)
    static constexpr int kRegs = HD > 128 ? 192 : 144, kLoaderRegs = HD > 128 ? 64 : 112;
    static_assert((kExactWarps * kRegs + kLoaders * kLoaderRegs) * 32 <= kThreads * 128, "registers of the launch");
    static constexpr int kParts = HD > 128 ? 4 : 1;  // a loader takes its rows of a stage in so many parts; kUnit: rows of one
    static constexpr int kUnit = kStage / (kLoaders * kParts);
    static constexpr int kLd = HD + 8;  // halves per row of a plane: eight rows hit different banks
    static constexpr int kPlane = kStage * kLd;
    // halves: planes (hi, lo) of q [kRows][kLd], of K [NB][kStage][kLd], of V; then floats: scales of q's, K's and V's rows
    static constexpr int kQ = 0, kK = 2 * kRows * kLd, kV = kK + 2 * NB * kPlane, kHalves = kV + 2 * NB * kPlane;
    static constexpr int kScaleQ = 0, kScaleK = kRows, kScaleV = kScaleK + NB * kStage;
    static constexpr int kProb = kScaleV + NB * kStage;  // a warp's probabilities
    static constexpr int kFloats = kProb + kExactWarps * 16 * TG;
    static constexpr size_t kOperands = 2 * static_cast<size_t>(kHalves) + 4 * kFloats;
    static constexpr size_t kFold = 4 * static_cast<size_t>(kExactNH * kRows * (HD + 4));  // per group: O and (m, l) of every row
    static constexpr size_t kBytes = (kOperands > kFold ? kOperands : kFold) + 16;
    static_assert(kBytes <= 227 * 1024, "shared memory of an SM");
    static_assert(kHalves % 8 == 0 && kProb % 4 == 0, "16-byte accesses");
};

// Two numbers as fp16 pairs hi + 2^-11 lo: 22 significant bits from 2^-14 on, 2^-36 off below it.  (Without the factor lo is out of normal
// numbers from 2^-3 on down.)
constexpr float kLoScale = 4.8828125e-4f;
__device__ __forceinline__ void splitPair(float a, float b, uint32_t &hi, uint32_t &lo) {
    hi = packHalf2(a, b);
    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
    const float2 r = __fmul2_rn(__ffma2_rn(f, make_float2(-1.0f, -1.0f), make_float2(a, b)), make_float2(2048.0f, 2048.0f));
    lo = packHalf2(r.x, r.y);
}
constexpr float kLeast = 6.103515625e-5f;  // 2^-14
// Rows in powers of two: `x`, the rows that a warp has in its hands (a unit), share one; scaled by it, their largest element is in
// [2^14, 2^15), and the pairs keep 22 bits of everything down to 2^-29 of that one and 2^-51 of it of what is smaller.  The bits of 2^e for a
// largest element in [2^e, 2^(e + 1)); infinities make it one.
template <int N, int NV>
__device__ __forceinline__ uint32_t unitExponent(const float4 (&x)[N][NV]) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int v = 0; v < NV; ++v) m = fmaxf(fmaxf(m, fmaxf(fabsf(x[i][v].x), fabsf(x[i][v].y))), fmaxf(fabsf(x[i][v].z), fabsf(x[i][v].w)));
    return max(__reduce_max_sync(0xffffffffu, __float_as_uint(m)) & 0x7f800000u, 15u << 23);
}
__device__ __forceinline__ float exactScale(uint32_t e) { return __uint_as_float((268u << 23) - e); }

// Where that is not enough: numbers in a unit below 2^-29 of its largest whose products with large ones elsewhere, or whose place in
// a dim of their own, let them count.  (One dim of 1e10 is no measure of the others.)  `low` follows the smallest |hi| that a lane has placed, NaN
// where one is; a unit with less than kLeast is looked at once more (inDoubt), for whether that was more than zeros (anySmall), and how many (isSmall).
__device__ __forceinline__ uint32_t leastOf(uint32_t a, uint32_t b) {  // magnitudes, the signs multiplied
    uint32_t r;
    asm("min.NaN.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ bool inDoubt(uint32_t low) {  // (warp-uniform)
    return __any_sync(0xffffffffu, !__hbge2(__habs2(*reinterpret_cast<const __half2 *>(&low)), __floats2half2_rn(kLeast, kLeast)));
}
template <int N, int NV>
__device__ __forceinline__ bool anySmall(const float4 (&x)[N][NV], uint32_t e, uint32_t low) {  // (warp-uniform)
    uint32_t m = 0xffffffffu;  // of what is not 0, the bits of the smallest magnitude, times two less one
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int v = 0; v < NV; ++v)
            m = min(min(min(m, 2u * __float_as_uint(x[i][v].x) - 1u), min(2u * __float_as_uint(x[i][v].y) - 1u, 2u * __float_as_uint(x[i][v].z) - 1u)),
                    2u * __float_as_uint(x[i][v].w) - 1u);
    const uint32_t least = max(max(e, 28u << 23) - (28u << 23), 1u);  // kLeast in the planes
    return __any_sync(0xffffffffu, m < 2u * least - 1u || (low & 0x7fffu) > 0x7c00u || (low >> 16 & 0x7fffu) > 0x7c00u);
}
__device__ __forceinline__ uint32_t isSmall(float x, float scale) {  // (one that is NaN: as many as make a unit's worth)
    return x == 0.0f || fabsf(x) * scale >= kLeast ? 0u : (x == x ? 1u : 16u);
}
__device__ __forceinline__ uint32_t isSmall(const float4 &x, float scale) {
    return isSmall(x.x, scale) + isSmall(x.y, scale) + isSmall(x.z, scale) + isSmall(x.w, scale);
}
template <int N, int NV>
__device__ __forceinline__ bool zeroDim(const float4 (&x)[N][NV]) {  // a dim that is 0 in all rows that a lane has of it (warp-uniform)
    bool zero = false;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < N; ++i)
            m.x = fmaxf(m.x, fabsf(x[i][v].x)), m.y = fmaxf(m.y, fabsf(x[i][v].y)), m.z = fmaxf(m.z, fabsf(x[i][v].z)), m.w = fmaxf(m.w, fabsf(x[i][v].w));
        zero = zero || m.x == 0.0f || m.y == 0.0f || m.z == 0.0f || m.w == 0.0f;
    }
    return __any_sync(0xffffffffu, zero);
}
// What a unit's scale says besides, for the warps that compute.  q, K: negative, it has small ones, which count when the score of
// such rows can be large (kSmallCount: HD x 2 x 2^15 x 2^-36 of that is 2^-24).  V: minus infinity, it has as many as it has rows: a
// dim of its own (fewer stay within 2^-51 of the unit's largest; N(0, 1) has one in 2 x 10^8); negative, a dim of it is zero, of which
// its weight says nothing: that counts where its scale is far from the others' (kLongScales).
constexpr float kSmallCount = 2.44140625e-4f, kMostScale = 1.2676506e30f;  // 2^-12; 2^100: a product with more might not fit
constexpr uint32_t kHugeWord = 240u << 23;   // a scale of q or K of 2^127 or an infinity
constexpr uint32_t kLongScales = 6u << 23;  // 2^6 of the first one's

// (what is worked out from it stays in the branch that asks for it, and out of the registers of the loop around)
__device__ __forceinline__ uint32_t opaqueZero() {
    uint32_t z;
    asm volatile("mov.u32 %0, 0;" : "=r"(z));
    return z;
}

// The token groups of a row put together: every warp's O (unnormalised), row maxima (log2 units) and row sums through
// shared memory, then out.  `out` is row 0 of the block, `ld` floats from row to row.
template <int HD>
__device__ __forceinline__ void exactFold(float *sm, const float (&o)[HD / 8][4], float m0, float m1, float l0, float l1,
                                          uint32_t nh, uint32_t rt, uint32_t rows, float *out, size_t ld) {
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
#pragma unroll
    for (int off = 1; off <= 2; off <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, off);
        l1 += __shfl_xor_sync(0xffffffffu, l1, off);
    }
    namedBarSync(kFoldBar, kExactThreads);  // the operands are done with: the fold's scratch takes their place
    float *scr = sm + (nh * kExactRows + rt * 16u + g) * (HD + 4);
#pragma unroll
    for (int d = 0; d < HD / 8; ++d) {
        *reinterpret_cast<float2 *>(scr + 8 * d + 2 * t) = make_float2(o[d][0], o[d][1]);
        *reinterpret_cast<float2 *>(scr + 8 * (HD + 4) + 8 * d + 2 * t) = make_float2(o[d][2], o[d][3]);
    }
    if (t == 0) {
        scr[HD] = m0, scr[HD + 1] = l0;
        scr[8 * (HD + 4) + HD] = m1, scr[8 * (HD + 4) + HD + 1] = l1;
    }
    namedBarSync(kFoldBar, kExactThreads);
    for (uint32_t i = threadIdx.x; i < rows * (HD / 4); i += kExactThreads) {
        const uint32_t r = i / (HD / 4), c = (i % (HD / 4)) * 4;
        const float *e = sm + r * (HD + 4);
        float M = kNegBig;
#pragma unroll
        for (int h = 0; h < kExactNH; ++h) M = fmaxf(M, e[h * kExactRows * (HD + 4) + HD]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float l = 0.0f;
#pragma unroll
        for (int h = 0; h < kExactNH; ++h) {
            const float *eh = e + h * kExactRows * (HD + 4);
            const float w = fastExp2(eh[HD] - M);
            l = fmaf(w, eh[HD + 1], l);
            const float4 a = *reinterpret_cast<const float4 *>(eh + c);
            acc.x = fmaf(w, a.x, acc.x);
            acc.y = fmaf(w, a.y, acc.y);
            acc.z = fmaf(w, a.z, acc.z);
            acc.w = fmaf(w, a.w, acc.w);
        }
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        *reinterpret_cast<float4 *>(out + r * ld + c) =
                make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    }
}

template <int HD>
__global__ void __launch_bounds__(ExactShape<HD>::kThreads, 1) prefillExactKernel(const __grid_constant__ PrefillExactParams p) {
    using S = ExactShape<HD>;
    constexpr int RT = kExactRT, TG = S::TG, LD = S::kLd, NT = TG / 8, NB = S::NB;
    constexpr uint32_t kAll = S::kThreads;
    constexpr uint32_t kFullK = kFoldBar + 1, kFullV = kFullK + NB, kFreeK = kFullV + NB, kFreeV = kFreeK + NB;  // named barriers per buffer
    constexpr int RW = HD < 128 ? 2 : 1, NV = HD > 128 ? 2 : 1;  // rows that a warp takes at a time, float4 per lane of them
    extern __shared__ __align__(16) float sm[];
    __half *sh = reinterpret_cast<__half *>(sm);
    float *sf = reinterpret_cast<float *>(sh + S::kHalves);
    gridDepWait();
    gridDepLaunch();

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t blk = gridDim.y - 1u - blockIdx.y, head = blockIdx.x;  // late rows (long prefixes) of all heads first
    const uint32_t row0 = blk * S::kRows, rows = min(static_cast<uint32_t>(S::kRows), p.qRows - row0);
    const uint32_t pos0 = p.devPos ? p.devPos[0] : p.cachePos;
    const uint64_t wanted = static_cast<uint64_t>(pos0) + row0 + rows;
    const uint32_t len = static_cast<uint32_t>(wanted < p.totalRows ? wanted : p.totalRows);  // (a device position past the store)
    const uint32_t nStages = (len + S::kStage - 1) / S::kStage;
    const uint32_t unit = HD < 128 ? lane % 16u : lane, sub = HD < 128 ? lane / 16u : 0u;  // this lane's float4 of a row, and which row
    // hi and lo parts of a piece of a row, into row r of the planes at `plane` (`lo` halves apart); `low` follows the smallest |hi|
    auto place = [&](__half *plane, uint32_t lo, const float4 (&x)[NV], float scale, uint32_t r, uint32_t &low) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            uint2 h, l;
            const float2 s2 = make_float2(scale, scale), a = __fmul2_rn(make_float2(x[v].x, x[v].y), s2), b = __fmul2_rn(make_float2(x[v].z, x[v].w), s2);
            splitPair(a.x, a.y, h.x, l.x);
            splitPair(b.x, b.y, h.y, l.y);
            low = leastOf(low, leastOf(h.x, h.y));
            __half *at = plane + r * LD + (unit + 32u * v) * 4u;
            *reinterpret_cast<uint2 *>(at) = h;
            *reinterpret_cast<uint2 *>(at + lo) = l;
        }
    };

    constexpr uint32_t kHighest = 0x7c007c00u;  // (infinities)

    if (warp >= kExactWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::kLoaderRegs));
        // ---- loaders: rows of a stage through registers into the planes, K and V in turn, the next ones on their way meanwhile ----
        constexpr uint32_t LW = S::kLoaders, H = S::kParts, NH = S::kUnit / RW;  // (float4s of a lane per unit: NH x NV)
        static_assert(NH * RW == S::kUnit && S::kUnit * H * LW == S::kStage, "even shares");
        const uint32_t lw = warp - kExactWarps, kvHead = head / p.group;
        const size_t stride = static_cast<size_t>(p.nKV) * (HD / 4);
        const float4 *gk = static_cast<const float4 *>(p.k) + static_cast<size_t>(kvHead) * (HD / 4);
        const float4 *gv = static_cast<const float4 *>(p.v) + static_cast<size_t>(kvHead) * (HD / 4);
        auto unitRow = [&](uint32_t part) { return (lw * H + part) * S::kUnit; };
        // (for rows behind the last one attended, that one: whatever is there meets probabilities of 0, and 0 x NaN would be NaN)
        auto load = [&](float4 (&x)[NH][NV], const float4 *src, uint32_t st, uint32_t part) {
            const uint32_t tok0 = st * S::kStage + unitRow(part) + sub;
            const float4 *at = src + tok0 * stride + unit;
            if ((st + 1u) * S::kStage <= len) {  // (a branch, not a condition per load)
#pragma unroll
                for (uint32_t i = 0; i < NH; ++i)
#pragma unroll
                    for (int v = 0; v < NV; ++v) x[i][v] = __ldg(at + i * (RW * stride) + 32u * v);
                return;
            }
#pragma unroll
            for (uint32_t i = 0; i < NH; ++i)
#pragma unroll
                for (int v = 0; v < NV; ++v) x[i][v] = __ldg(src + min(tok0 + i * RW, len - 1u) * stride + unit + 32u * v);
        };
        auto put = [&](const float4 (&x)[NH][NV], __half *plane, uint32_t *scales, uint32_t st, uint32_t part, bool isV) {
            const uint32_t e = unitExponent<NH, NV>(x), row = unitRow(part);
            const float scale = exactScale(e);
            uint32_t low = kHighest;
#pragma unroll
            for (uint32_t i = 0; i < NH; ++i) place(plane, S::kPlane, x[i], scale, row + i * RW + sub, low);
            uint32_t word = isV ? e : e - (14u << 23);  // V: 2^e, the probabilities carry it; K: what undoes the scale
            if (lane < S::kUnit) scales[row + lane] = word;
            if (inDoubt(low)) {
                if (isV && e > (15u << 23) && zeroDim<NH, NV>(x)) word |= 0x80000000u;  // (a unit of nothing but zeros weighs nothing)
                if (anySmall<NH, NV>(x, e, low)) {
                    uint32_t small = 0u;
#pragma unroll 1
                    for (uint32_t i = opaqueZero(); i < NH; ++i)
#pragma unroll
                        for (int v = 0; v < NV; ++v)
                            small += isSmall(__ldg((isV ? gv : gk) + min(st * S::kStage + row + i * RW + sub, len - 1u) * stride + unit + 32u * v), scale);
                    small = __reduce_add_sync(0xffffffffu, small);
                    word = isV ? (small >= S::kUnit ? 0xff800000u : word) : word | 0x80000000u;
                }
                if (lane < S::kUnit) scales[row + lane] = word;
            }
        };
        if (nStages == 0u) return;  // (an empty store)
        // parts in turn: those of K, those of V; two are on their way
        float4 x[2][NH][NV];
        load(x[0], gk, 0, 0);
        load(x[1], H == 1 ? gv : gk, 0, H == 1 ? 0 : 1);
        for (uint32_t st = 0; st < nStages; ++st) {
            const uint32_t buf = st % NB;
            __half *planes[2] = {sh + S::kK + buf * 2 * S::kPlane, sh + S::kV + buf * 2 * S::kPlane};
            uint32_t *scales[2] = {reinterpret_cast<uint32_t *>(sf + S::kScaleK + buf * S::kStage), reinterpret_cast<uint32_t *>(sf + S::kScaleV + buf * S::kStage)};
#pragma unroll
            for (uint32_t j = 0; j < 2 * H; ++j) {
                const bool isV = j >= H;
                if (j % H == 0 && st >= NB) namedBarSync((isV ? kFreeV : kFreeK) + buf, kAll);
                put(x[j & 1u], planes[isV], scales[isV], st, j % H, isV);
                const uint32_t next = j + 2, nextSt = st + next / (2 * H), part = next % (2 * H);
                if (nextSt < nStages) load(x[j & 1u], part >= H ? gv : gk, nextSt, part % H);
                if (j % H == H - 1) namedBarArrive((isV ? kFullV : kFullK) + buf, kAll);
            }
        }
        return;
    }

    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::kRegs));
    const uint32_t g = lane >> 2, t = lane & 3u, rt = warp % RT, nh = warp / RT;
    {   // q, the same way
        constexpr uint32_t N = S::kRows / (kExactWarps * RW);
        float4 x[N][NV];
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const uint32_t r = min((i * kExactWarps + warp) * RW + sub, rows - 1u);  // (no row: the last one)
#pragma unroll
            for (int v = 0; v < NV; ++v)
                x[i][v] = __ldg(reinterpret_cast<const float4 *>(p.q + (static_cast<size_t>(row0 + r) * p.nHeads + head) * HD) + unit + 32u * v);
        }
        const uint32_t e = unitExponent<N, NV>(x);
        const float scale = exactScale(e);
        uint32_t low = kHighest, word = e - (14u << 23);
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) place(sh + S::kQ, S::kRows * LD, x[i], scale, (i * kExactWarps + warp) * RW + sub, low);
        if (inDoubt(low) && anySmall<N, NV>(x, e, low)) word |= 0x80000000u;
        if (unit == 0) {
#pragma unroll
            for (uint32_t i = 0; i < N; ++i) sf[S::kScaleQ + (i * kExactWarps + warp) * RW + sub] = __uint_as_float(word);
        }
    }
    namedBarSync(kFoldBar, kExactThreads);
    const float cs0 = p.scaleLog2 * fabsf(sf[S::kScaleQ + rt * 16u + g]), cs1 = p.scaleLog2 * fabsf(sf[S::kScaleQ + rt * 16u + g + 8u]);
    // the largest scale of this warp's rows, whether they have small ones, and from where on a word of K's is looked into (a sign above all)
    uint32_t csTop, kDoubt;
    bool qSmall;
    {
        const uint32_t word = __float_as_uint(sf[S::kScaleQ + rt * 16u + (lane & 15u)]);
        qSmall = __any_sync(0xffffffffu, word >> 31);
        const uint32_t top = __reduce_max_sync(0xffffffffu, word & 0x7fffffffu);
        csTop = top < kHugeWord ? __float_as_uint(fabsf(p.scaleLog2) * __uint_as_float(top)) : 0x7f800000u;
        kDoubt = qSmall || top >= kHugeWord ? 0u : min(max(354u - (csTop >> 23), 1u), kHugeWord >> 23) << 23;  // (2^99 or 2^100 with csTop)
    }

    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    float m0 = kNegBig, m1 = kNegBig, l0 = 0.0f, l1 = 0.0f;
    // this thread's query rows (g and g + 8 of the warp's tile) see tokens below (with a device position past the store, the rows there are):
    const uint32_t lim0 = min(len, pos0 + row0 + rt * 16u + g + 1u), lim1 = min(len, pos0 + row0 + rt * 16u + g + 9u);
    const uint32_t warpLimit = min(len, pos0 + row0 + rt * 16u + 16u);  // no row of the warp's tile sees further

    // ldmatrix: lane i delivers row i % 8 of 8x8 block i / 8
    const uint32_t aAddr = smemAddr(sh + S::kQ + (rt * 16u + (lane & 15u)) * LD + (lane >> 4) * 8u);
    // K: blocks (tokens 0-7, dims 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15)
    const uint32_t kAddr = smemAddr(sh + S::kK + (nh * TG + (lane & 7u) + (lane >> 4) * 8u) * LD + ((lane >> 3) & 1u) * 8u);
    // V, transposed: blocks (tokens 0-7, dims 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
    const uint32_t vAddr = smemAddr(sh + S::kV + (nh * TG + (lane & 15u)) * LD + (lane >> 4) * 8u);
    constexpr uint32_t kLoAt = S::kPlane * 2, kBufAt = 2 * kLoAt;  // bytes

    float s[NT][4];
    // scores (log2 units) to probabilities: this thread has tokens 2t, 2t + 1 of every 8, rows g and g + 8
    constexpr int NU = S::kUnit < 8 ? 1 : TG / S::kUnit;  // a group's units with a largest probability each (smaller ones do it without)
    float pm0[NU], pm1[NU];
    auto softmax = [&](uint32_t tok0, uint32_t freeK, bool again) {
        float mu0[NU], mu1[NU];
#pragma unroll
        for (int u = 0; u < NU; ++u) mu0[u] = mu1[u] = kNegBig;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t tok = tok0 + 8 * n + 2 * t + i;
                s[n][i] = tok < lim0 ? s[n][i] : -INFINITY;
                s[n][2 + i] = tok < lim1 ? s[n][2 + i] : -INFINITY;
                mu0[n * NU / NT] = fmaxf(mu0[n * NU / NT], s[n][i]);
                mu1[n * NU / NT] = fmaxf(mu1[n * NU / NT], s[n][2 + i]);
            }
        __syncwarp();  // (every lane has read its part of K and of its scales)
        if (again) namedBarArrive(freeK, kAll);
        float mn0 = m0, mn1 = m1;
#pragma unroll
        for (int u = 0; u < NU; ++u) {
#pragma unroll
            for (int off = 1; off <= 2; off <<= 1) {
                mu0[u] = fmaxf(mu0[u], __shfl_xor_sync(0xffffffffu, mu0[u], off));
                mu1[u] = fmaxf(mu1[u], __shfl_xor_sync(0xffffffffu, mu1[u], off));
            }
            mn0 = fmaxf(mn0, mu0[u]), mn1 = fmaxf(mn1, mu1[u]);
        }
        if (__any_sync(0xffffffffu, mn0 != m0 || mn1 != m1)) {
            const float a0 = fastExp2(m0 - mn0), a1 = fastExp2(m1 - mn1);
#pragma unroll
            for (int i = 0; i < HD / 8; ++i) {
                o[i][0] *= a0;
                o[i][1] *= a0;
                o[i][2] *= a1;
                o[i][3] *= a1;
            }
            l0 *= a0;
            l1 *= a1;
            m0 = mn0;
            m1 = mn1;
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            s[n][0] = fastExp2(s[n][0] - m0), s[n][1] = fastExp2(s[n][1] - m0);
            s[n][2] = fastExp2(s[n][2] - m1), s[n][3] = fastExp2(s[n][3] - m1);
            l0 += s[n][0] + s[n][1];
            l1 += s[n][2] + s[n][3];
        }
#pragma unroll
        for (int u = 0; u < NU; ++u) pm0[u] = fastExp2(mu0[u] - m0), pm1[u] = fastExp2(mu1[u] - m1);
    };

    uint32_t st = 0, at = 0;  // (at: how far the stage is that did not fit -- 1: its K is in, 2: its probabilities and V are)
    for (; st < nStages; ++st) {
        const uint32_t buf = st % NB, tok0 = st * S::kStage + nh * TG;
        const bool active = tok0 < warpLimit, again = st + NB < nStages;  // (both warp-uniform)
        namedBarSync(kFullK + buf, kAll);
        if (active) {
            const float *sk = sf + S::kScaleK + buf * S::kStage + nh * TG;
            const uint32_t word = __float_as_uint(sk[lane % TG]);
            float x[NT][4];  // s: hi*hi, x: the cross terms
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] = x[n][i] = 0.0f;
#pragma unroll(HD == 64 ? 4 : 2)
            for (int ks = 0; ks < HD / 16; ++ks) {
                uint32_t ah[4], al[4], bh[NT / 2][4], bl[NT / 2][4];
                ldmatrixX4(ah[0], ah[1], ah[2], ah[3], aAddr + ks * 32);
                ldmatrixX4(al[0], al[1], al[2], al[3], aAddr + S::kRows * LD * 2 + ks * 32);
#pragma unroll
                for (int n = 0; n < NT / 2; ++n) {
                    const uint32_t from = kAddr + buf * kBufAt + n * (16 * LD * 2) + ks * 32;
                    ldmatrixX4(bh[n][0], bh[n][1], bh[n][2], bh[n][3], from);
                    ldmatrixX4(bl[n][0], bl[n][1], bl[n][2], bl[n][3], from + kLoAt);
                }
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(s[n], ah[0], ah[1], ah[2], ah[3], bh[n / 2][n % 2 * 2], bh[n / 2][n % 2 * 2 + 1]);
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(x[n], al[0], al[1], al[2], al[3], bh[n / 2][n % 2 * 2], bh[n / 2][n % 2 * 2 + 1]);
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(x[n], ah[0], ah[1], ah[2], ah[3], bl[n / 2][n % 2 * 2], bl[n / 2][n % 2 * 2 + 1]);
            }
            if (__any_sync(0xffffffffu, word >= kDoubt)) {  // (here the vote is no wait)
                const float top = __uint_as_float(word & 0x7fffffffu) * __uint_as_float(csTop);
                const bool holds = top <= kMostScale && (word & 0x7fffffffu) < kHugeWord && !((word >> 31 || qSmall) && top > kSmallCount);
                if (!__all_sync(0xffffffffu, holds)) {
                    at = 1;
                    break;
                }
            }
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float2 w = *reinterpret_cast<const float2 *>(sk + 8 * n + 2 * t);
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] = fmaf(x[n][i], kLoScale, s[n][i]) * (fabsf(i & 1 ? w.y : w.x) * (i & 2 ? cs1 : cs0));
            }
            softmax(tok0, kFreeK + buf, again);
        } else if (again) {
            namedBarArrive(kFreeK + buf, kAll);
        }
        namedBarSync(kFullV + buf, kAll);
        if (active) {
            // ---- O += P V, 16 tokens at a time: the accumulator layout of the scores is the A operand's.  The probabilities take the
            // scales of V's units along, and every query row a power of two of its own: the most that one of its products can be ----
            const float *sv = sf + S::kScaleV + buf * S::kStage + nh * TG;
            const uint32_t word = __float_as_uint(sv[lane % TG]);
            const bool doubt = __any_sync(0xffffffffu, word >= 0x7f800000u);
            float top0 = 0.0f, top1 = 0.0f, u[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float2 w = *reinterpret_cast<const float2 *>(sv + 8 * n + 2 * t);
#pragma unroll
                for (int i = 0; i < 4; ++i) u[n][i] = s[n][i] * fabsf(i & 1 ? w.y : w.x);
                if constexpr (S::kUnit >= 8) {  // (w is the same for all of a unit)
                    top0 = fmaxf(top0, pm0[n * NU / NT] * fabsf(w.x));
                    top1 = fmaxf(top1, pm1[n * NU / NT] * fabsf(w.x));
                } else {
                    top0 = fmaxf(top0, fmaxf(u[n][0], u[n][1]));
                    top1 = fmaxf(top1, fmaxf(u[n][2], u[n][3]));
                }
            }
            if constexpr (S::kUnit < 8) {
#pragma unroll
                for (int off = 1; off <= 2; off <<= 1) {
                    top0 = fmaxf(top0, __shfl_xor_sync(0xffffffffu, top0, off));
                    top1 = fmaxf(top1, __shfl_xor_sync(0xffffffffu, top1, off));
                }
            }
            const uint32_t e0 = max(__float_as_uint(top0) & 0x7f800000u, 15u << 23), e1 = max(__float_as_uint(top1) & 0x7f800000u, 15u << 23);
            const float in0 = exactScale(e0), in1 = exactScale(e1);
            if (doubt) {
                bool holds = true;
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) holds = holds && !(u[n][i] != 0.0f && u[n][i] * (i & 2 ? in1 : in0) < kLeast);
                const uint32_t scale = word & 0x7fffffffu, first = __float_as_uint(sv[0]) & 0x7fffffffu;
                const bool near = !__any_sync(0xffffffffu, scale - first + kLongScales > 2u * kLongScales);
                holds = (holds || near) && scale < 0x7f800000u;
                if (!__all_sync(0xffffffffu, holds)) {
                    at = 2;
                    break;
                }
            }
            uint32_t ph[NT / 2][4], pl[NT / 2][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                splitPair(u[n][0] * in0, u[n][1] * in0, ph[n / 2][n % 2 * 2], pl[n / 2][n % 2 * 2]);
                splitPair(u[n][2] * in1, u[n][3] * in1, ph[n / 2][n % 2 * 2 + 1], pl[n / 2][n % 2 * 2 + 1]);
            }
            constexpr float kPlanes = 3.7252902984619140625e-9f;  // 2^-28: 2^14 in the planes of V, and in the pairs of p
            const float out0 = __uint_as_float(e0) * kPlanes, out1 = __uint_as_float(e1) * kPlanes;
            constexpr int DB = HD > 128 ? 1 : 2;  // pairs of dim tiles at a time, their chains alternating
#pragma unroll
            for (int d0 = 0; d0 < HD / 16; d0 += DB) {
                float sum[2 * DB][4] = {}, cross[2 * DB][4] = {};  // a stage's products by themselves (see the head of the file)
#pragma unroll
                for (int n = 0; n < NT / 2; ++n) {
                    uint32_t bh[DB][4], bl[DB][4];
#pragma unroll
                    for (int d = 0; d < DB; ++d) {
                        const uint32_t from = vAddr + buf * kBufAt + n * (16 * LD * 2) + (d0 + d) * 32;
                        ldmatrixX4Trans(bh[d][0], bh[d][1], bh[d][2], bh[d][3], from);
                        ldmatrixX4Trans(bl[d][0], bl[d][1], bl[d][2], bl[d][3], from + kLoAt);
                    }
#pragma unroll
                    for (int d = 0; d < 2 * DB; ++d)
                        mmaF16(sum[d], ph[n][0], ph[n][1], ph[n][2], ph[n][3], bh[d / 2][d % 2 * 2], bh[d / 2][d % 2 * 2 + 1]);
#pragma unroll
                    for (int d = 0; d < 2 * DB; ++d)
                        mmaF16(cross[d], pl[n][0], pl[n][1], pl[n][2], pl[n][3], bh[d / 2][d % 2 * 2], bh[d / 2][d % 2 * 2 + 1]);
#pragma unroll
                    for (int d = 0; d < 2 * DB; ++d)
                        mmaF16(cross[d], ph[n][0], ph[n][1], ph[n][2], ph[n][3], bl[d / 2][d % 2 * 2], bl[d / 2][d % 2 * 2 + 1]);
                }
#pragma unroll
                for (int d = 0; d < 2 * DB; ++d)
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[2 * d0 + d][i] = fmaf(fmaf(cross[d][i], kLoScale, sum[d][i]), i & 2 ? out1 : out0, o[2 * d0 + d][i]);
            }
            __syncwarp();
        }
        if (again) namedBarArrive(kFreeV + buf, kAll);
    }

    // From the first stage on whose numbers the pairs do not hold: the same in f32, from the rows themselves, hand in hand with the loaders
    // still.  (In the loop above it cost every stage 4 - 6 %.)
    for (; st < nStages; ++st, at = 0) {
        const uint32_t buf = st % NB, tok0 = st * S::kStage + nh * TG;
        const bool active = tok0 < warpLimit, again = st + NB < nStages;
        if (at == 0) namedBarSync(kFullK + buf, kAll);
        if (at < 2) {
            if (active) {
                const float4 *qa = reinterpret_cast<const float4 *>(p.q + (static_cast<size_t>(row0 + min(rt * 16u + g, rows - 1u)) * p.nHeads + head) * HD);
                const float4 *qb = reinterpret_cast<const float4 *>(p.q + (static_cast<size_t>(row0 + min(rt * 16u + g + 8u, rows - 1u)) * p.nHeads + head) * HD);
                const float4 *gk = static_cast<const float4 *>(p.k) + static_cast<size_t>(head / p.group) * (HD / 4);
                float x[NT][4];
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[n][i] = x[n][i] = 0.0f;
#pragma unroll 1
                for (uint32_t c = 0; c < HD / 4; ++c) {
                    const float4 a = __ldg(qa + c), b = __ldg(qb + c);
#pragma unroll
                    for (int n = 0; n < NT; ++n)
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t tok = min(tok0 + 8 * n + 2 * t + i, len - 1u);
                            const float4 k = __ldg(gk + static_cast<size_t>(tok) * p.nKV * (HD / 4) + c);
                            s[n][i] = fmaf(a.x, k.x, fmaf(a.y, k.y, s[n][i])), x[n][i] = fmaf(a.z, k.z, fmaf(a.w, k.w, x[n][i]));
                            s[n][2 + i] = fmaf(b.x, k.x, fmaf(b.y, k.y, s[n][2 + i])), x[n][2 + i] = fmaf(b.z, k.z, fmaf(b.w, k.w, x[n][2 + i]));
                        }
                }
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[n][i] = (s[n][i] + x[n][i]) * p.scaleLog2;
                softmax(tok0, kFreeK + buf, again);
            } else if (again) {
                namedBarArrive(kFreeK + buf, kAll);
            }
            namedBarSync(kFullV + buf, kAll);
        }
        if (active) {
            // the warp's probabilities through shared memory: a thread takes all tokens of its two rows for the dims it has
            float *prob = sf + S::kProb + warp * 16 * TG;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                *reinterpret_cast<float2 *>(prob + g * TG + 8 * n + 2 * t) = make_float2(s[n][0], s[n][1]);
                *reinterpret_cast<float2 *>(prob + (g + 8u) * TG + 8 * n + 2 * t) = make_float2(s[n][2], s[n][3]);
            }
            __syncwarp();
            const float2 *gv = static_cast<const float2 *>(p.v) + static_cast<size_t>(head / p.group) * (HD / 2) + t;
#pragma unroll 1
            for (uint32_t c = 0; c < TG && tok0 + c < warpLimit; ++c) {
                const float p0 = prob[g * TG + c], p1 = prob[(g + 8u) * TG + c];
                const bool see0 = tok0 + c < lim0, see1 = tok0 + c < lim1;  // (masked rows stay out: 0 x Inf would be NaN)
                const float2 *row = gv + static_cast<size_t>(tok0 + c) * p.nKV * (HD / 2);
#pragma unroll
                for (int d = 0; d < HD / 8; ++d) {
                    const float2 v = __ldg(row + 4 * d);
                    if (see0) o[d][0] = fmaf(p0, v.x, o[d][0]), o[d][1] = fmaf(p0, v.y, o[d][1]);
                    if (see1) o[d][2] = fmaf(p1, v.x, o[d][2]), o[d][3] = fmaf(p1, v.y, o[d][3]);
                }
            }
            __syncwarp();
        }
        if (again) namedBarArrive(kFreeV + buf, kAll);
    }
    exactFold<HD>(sm, o, m0, m1, l0, l1, nh, rt, rows, p.out + (static_cast<size_t>(row0) * p.nHeads + head) * HD,
                  static_cast<size_t>(p.nHeads) * HD);
}

// ---- fp16 store ------------------------------------------------------------------------------------------
// fp16 K and V are operands as they are, in one plane each and two products where the f32 rows need three; q, normalised by
// a power of two per row, and the probabilities are fp16 hi + lo pairs (two products, ~22 mantissa bits), as in
// decode_kv16.cu.  Stages come in by cp.async, two deep.
template <int HD>
struct ExactHalfShape {
    static constexpr int TG = 32, BPS = HD == 64 ? 2 : 1, kRows = kExactRows, kStage = kExactNH * TG, kThreads = kExactThreads;
    static constexpr int kLd = HD + 8;                       // halves per row: eight rows hit different banks
    static constexpr int kQ = 0;                             // q hi, lo [kRows][kLd]
    static constexpr int kKV = 2 * kRows * kLd;              // [2 stages][K, V][kStage][kLd]
    static constexpr int kHalves = kKV + 4 * kStage * kLd;
    static constexpr int kFold = 2 * kExactNH * kRows * (HD + 4);  // in halves
    static constexpr size_t kBytes = 2 * static_cast<size_t>(kHalves > kFold ? kHalves : kFold) + 16;
    static_assert(kBytes * BPS <= 227 * 1024, "shared memory of an SM");
};

template <int HD>
__global__ void __launch_bounds__(kExactThreads, ExactHalfShape<HD>::BPS)
prefillExactHalfKernel(const __grid_constant__ PrefillExactParams p) {
    using S = ExactHalfShape<HD>;
    constexpr int RT = kExactRT, TG = S::TG, LD = S::kLd, NT = TG / 8;
    constexpr uint32_t kThreads = kExactWarps * 32, U = HD / 8;  // 16-byte units per row
    extern __shared__ __align__(16) float sm[];
    __half *sh = reinterpret_cast<__half *>(sm);
    __shared__ float sScale[S::kRows];  // log2-domain scale of a row's products
    gridDepWait();
    gridDepLaunch();

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t rt = warp % RT, nh = warp / RT;
    const uint32_t blk = gridDim.y - 1u - blockIdx.y, head = blockIdx.x;  // late rows (long prefixes) of all heads first
    const uint32_t row0 = blk * S::kRows, rows = min(static_cast<uint32_t>(S::kRows), p.qRows - row0);
    const uint32_t pos0 = p.devPos ? p.devPos[0] : p.cachePos;
    const uint64_t wanted = static_cast<uint64_t>(pos0) + row0 + rows;
    const uint32_t len = static_cast<uint32_t>(wanted < p.totalRows ? wanted : p.totalRows);
    const uint32_t kvHead = head / p.group;

    const uint4 *gk = static_cast<const uint4 *>(p.k) + static_cast<size_t>(kvHead) * U;
    const uint4 *gv = static_cast<const uint4 *>(p.v) + static_cast<size_t>(kvHead) * U;
    const size_t stride = static_cast<size_t>(p.nKV) * U;
    const uint32_t kv0 = smemAddr(sh + S::kKV);
    auto request = [&](uint32_t st) {
        const uint32_t base = kv0 + (st & 1u) * (2 * S::kStage * LD * 2), tok0 = st * S::kStage;
        for (uint32_t i = threadIdx.x; i < S::kStage * U; i += kThreads) {
            const uint32_t r = i / U, c = i % U, ok = tok0 + r < len ? 16u : 0u;  // rows behind the last one are zeros
            const size_t at = ok ? (tok0 + r) * stride + c : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + (r * LD + c * 8) * 2), "l"(gk + at), "r"(ok) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + ((S::kStage + r) * LD + c * 8) * 2), "l"(gv + at),
                         "r"(ok) : "memory");
        }
        cpAsyncCommit();
    };
    const uint32_t nStages = (len + S::kStage - 1) / S::kStage;
    {   // q: HD / 4 lanes per row; its loads go ahead of the first stages' copies, or they queue behind them
        constexpr uint32_t W = HD / 4, R = 32 / W, N = S::kRows / (kExactWarps * R);
        static_assert(S::kRows % (kExactWarps * R) == 0, "even shares");
        float4 qv[N];
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const uint32_t r = (i * kExactWarps + warp) * R + lane / W, c = lane % W * 4;
            qv[i] = r < rows ? *reinterpret_cast<const float4 *>(p.q + (static_cast<size_t>(row0 + r) * p.nHeads + head) * HD + c)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        request(0);
        if (nStages > 1) request(1);
        else cpAsyncCommit();
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const uint32_t r = (i * kExactWarps + warp) * R + lane / W, c = lane % W * 4;
            const float4 x = qv[i];
            float amax = fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w)));
#pragma unroll
            for (int o = W / 2; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            int e = static_cast<int>((__float_as_uint(amax) >> 23) & 0xffu) - 127;  // floor(log2 amax)
            e = amax > 0.0f ? max(-100, min(100, e)) : 0;
            const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
            float h[4], l[4];
            splitHalf(x.x * down, h[0], l[0]);
            splitHalf(x.y * down, h[1], l[1]);
            splitHalf(x.z * down, h[2], l[2]);
            splitHalf(x.w * down, h[3], l[3]);
            *reinterpret_cast<uint2 *>(sh + r * LD + c) = make_uint2(packHalf2(h[0], h[1]), packHalf2(h[2], h[3]));
            *reinterpret_cast<uint2 *>(sh + (S::kRows + r) * LD + c) = make_uint2(packHalf2(l[0], l[1]), packHalf2(l[2], l[3]));
            if (c == 0) sScale[r] = p.scaleLog2 * __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
        }
    }

    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    float m0 = kNegBig, m1 = kNegBig, l0 = 0.0f, l1 = 0.0f;
    const uint32_t lim0 = pos0 + row0 + rt * 16u + g + 1u, lim1 = lim0 + 8u;
    const uint32_t warpLimit = min(len, pos0 + row0 + rt * 16u + 16u);
    // ldmatrix: lane i delivers row i % 8 of 8x8 block i / 8
    const uint32_t aAddr = smemAddr(sh + (rt * 16u + (lane & 15u)) * LD + (lane >> 4) * 8u);
    // K: blocks (tokens 0-7, dims 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15)
    const uint32_t kOff = ((nh * TG + (lane & 7u) + (lane >> 4) * 8u) * LD + ((lane >> 3) & 1u) * 8u) * 2;
    // V, transposed: blocks (tokens 0-7, dims 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
    const uint32_t vOff = ((S::kStage + nh * TG + (lane & 15u)) * LD + (lane >> 4) * 8u) * 2;
    float cs0 = 0.0f, cs1 = 0.0f;

    for (uint32_t st = 0; st < nStages; ++st) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // the stage is in for everybody (and, the first time, q is)
        if (st == 0) cs0 = sScale[rt * 16u + g], cs1 = sScale[rt * 16u + g + 8u];
        const uint32_t base = kv0 + (st & 1u) * (2 * S::kStage * LD * 2);
        const uint32_t tok0 = st * S::kStage + nh * TG;
        if (tok0 < warpLimit) {  // warp-uniform
            float s[NT][4], x[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] = x[n][i] = 0.0f;
#pragma unroll 4
            for (int ks = 0; ks < HD / 16; ++ks) {
                uint32_t ah[4], al[4], b[NT / 2][4];
                ldmatrixX4(ah[0], ah[1], ah[2], ah[3], aAddr + ks * 32);
                ldmatrixX4(al[0], al[1], al[2], al[3], aAddr + S::kRows * LD * 2 + ks * 32);
#pragma unroll
                for (int n = 0; n < NT / 2; ++n)
                    ldmatrixX4(b[n][0], b[n][1], b[n][2], b[n][3], base + kOff + n * (16 * LD * 2) + ks * 32);
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(s[n], ah[0], ah[1], ah[2], ah[3], b[n / 2][n % 2 * 2], b[n / 2][n % 2 * 2 + 1]);
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(x[n], al[0], al[1], al[2], al[3], b[n / 2][n % 2 * 2], b[n / 2][n % 2 * 2 + 1]);
            }
            float mx0 = kNegBig, mx1 = kNegBig;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t tok = tok0 + 8 * n + 2 * t + i;
                    s[n][i] = tok < lim0 ? (s[n][i] + x[n][i]) * cs0 : -INFINITY;
                    s[n][2 + i] = tok < lim1 ? (s[n][2 + i] + x[n][2 + i]) * cs1 : -INFINITY;
                    mx0 = fmaxf(mx0, s[n][i]);
                    mx1 = fmaxf(mx1, s[n][2 + i]);
                }
#pragma unroll
            for (int off = 1; off <= 2; off <<= 1) {
                mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
                mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
            }
            const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
            if (__any_sync(0xffffffffu, mn0 != m0 || mn1 != m1)) {
                const float a0 = fastExp2(m0 - mn0), a1 = fastExp2(m1 - mn1);
#pragma unroll
                for (int i = 0; i < HD / 8; ++i) {
                    o[i][0] *= a0;
                    o[i][1] *= a0;
                    o[i][2] *= a1;
                    o[i][3] *= a1;
                }
                l0 *= a0;
                l1 *= a1;
                m0 = mn0;
                m1 = mn1;
            }
            // 16 tokens at a time: the accumulator layout of the scores is the A operand's
            uint32_t ph[NT / 2][4], pl[NT / 2][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float h[4], l[4];
                const float p0 = fastExp2(s[n][0] - m0), p1 = fastExp2(s[n][1] - m0);
                const float p2 = fastExp2(s[n][2] - m1), p3 = fastExp2(s[n][3] - m1);
                l0 += p0 + p1;
                l1 += p2 + p3;
                splitHalf(p0, h[0], l[0]);
                splitHalf(p1, h[1], l[1]);
                splitHalf(p2, h[2], l[2]);
                splitHalf(p3, h[3], l[3]);
                const int k = n % 2;
                ph[n / 2][2 * k] = packHalf2(h[0], h[1]), ph[n / 2][2 * k + 1] = packHalf2(h[2], h[3]);
                pl[n / 2][2 * k] = packHalf2(l[0], l[1]), pl[n / 2][2 * k + 1] = packHalf2(l[2], l[3]);
            }
            constexpr int DB = HD == 64 ? 2 : 4;  // pairs of dim tiles at a time, their chains alternating
#pragma unroll
            for (int d0 = 0; d0 < HD / 16; d0 += DB) {
                float sum[2 * DB][4] = {};  // a stage's products by themselves (see the head of the file)
#pragma unroll
                for (int n = 0; n < NT / 2; ++n) {
                    uint32_t b[DB][4];
#pragma unroll
                    for (int d = 0; d < DB; ++d)
                        ldmatrixX4Trans(b[d][0], b[d][1], b[d][2], b[d][3], base + vOff + n * (16 * LD * 2) + (d0 + d) * 32);
#pragma unroll
                    for (int d = 0; d < 2 * DB; ++d)
                        mmaF16(sum[d], pl[n][0], pl[n][1], pl[n][2], pl[n][3], b[d / 2][d % 2 * 2], b[d / 2][d % 2 * 2 + 1]);
#pragma unroll
                    for (int d = 0; d < 2 * DB; ++d)
                        mmaF16(sum[d], ph[n][0], ph[n][1], ph[n][2], ph[n][3], b[d / 2][d % 2 * 2], b[d / 2][d % 2 * 2 + 1]);
                }
#pragma unroll
                for (int d = 0; d < 2 * DB; ++d)
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[2 * d0 + d][i] += sum[d][i];
            }
        }
        __syncthreads();  // everybody is through with the stage
        if (st + 2 < nStages) request(st + 2);
        else cpAsyncCommit();
    }
    exactFold<HD>(sm, o, m0, m1, l0, l1, nh, rt, rows,
                                                   p.out + (static_cast<size_t>(row0) * p.nHeads + head) * HD,
                                                   static_cast<size_t>(p.nHeads) * HD);
}

template <typename S, typename K>
static int launchExact(K kern, bool (&attrDone)[64], const PrefillExactParams &prm, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attrDone[dev]) {
        TC_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(S::kBytes)));
        attrDone[dev] = true;
    }
    return launchDependent(kern, dim3(prm.nHeads, (prm.qRows + kExactRows - 1) / kExactRows), S::kThreads, S::kBytes, st, 1, prm);
}
template <int HD>
static int exact32(const PrefillExactParams &prm, cudaStream_t st) {
    static bool done[64] = {false};
    return launchExact<ExactShape<HD>>(prefillExactKernel<HD>, done, prm, st);
}
template <int HD>
static int exact16(const PrefillExactParams &prm, cudaStream_t st) {
    static bool done[64] = {false};
    return launchExact<ExactHalfShape<HD>>(prefillExactHalfKernel<HD>, done, prm, st);
}

// Which form a launch takes.  A block of the 8-row form (12 to 16 warps, each with tiles of its own) goes through a prefix
// two to four times faster than a 32-row block, but there are four times as many of them.  Both fill an SM, so a launch
// takes waves x (what a block costs at its ends + tokens x what one costs it), and at least what its longest block does.
// Microseconds, from 2 to 2000 rows behind 0 to 8000:
struct ExactCost {
    float end8, token8, end32, token32;
};
bool prefillExactWins(uint32_t rows, uint64_t before, uint32_t nHeads, uint32_t hd, int kvHalf) {
    static constexpr ExactCost k32[3] = {{3.0f, 0.0103f, 3.7f, 0.0174f}, {4.2f, 0.0193f, 3.8f, 0.038f}, {5.1f, 0.0548f, 5.8f, 0.069f}};
    static constexpr ExactCost k16[2] = {{3.4f, 0.0032f, 2.9f, 0.0115f}, {4.8f, 0.0049f, 4.3f, 0.019f}};
    const ExactCost &c = kvHalf ? k16[hd == 128] : k32[hd == 64 ? 0 : (hd == 128 ? 1 : 2)];
    const float last = static_cast<float>(before + rows), mean = static_cast<float>(before) + 0.5f * rows;
    const uint64_t sms = static_cast<uint64_t>(numSMs());
    auto us = [&](uint32_t blockRows, float end, float token) {
        const uint64_t blocks = static_cast<uint64_t>((rows + blockRows - 1) / blockRows) * nHeads;
        const float waves = static_cast<float>((blocks + sms - 1) / sms);
        return fmaxf(end + token * last, waves * (end + token * mean));
    };
    return us(32, c.end32, c.token32) < us(8, c.end8, c.token8);
}

// Arguments validated by the caller (decode_kv.cu).
int prefillExact(const float *q, const void *kvK, const void *kvV, float *out, uint32_t seqLen, uint32_t nHeads,
                 uint32_t nKV, uint32_t hd, uint32_t cachePos, const uint32_t *devPos, uint64_t totalRows, float invSqrt,
                 int kvHalf, cudaStream_t st) {
    PrefillExactParams prm;
    prm.q = q, prm.out = out, prm.k = kvK, prm.v = kvV;
    prm.devPos = devPos, prm.totalRows = totalRows;
    prm.qRows = seqLen, prm.cachePos = cachePos, prm.nHeads = nHeads, prm.nKV = nKV, prm.group = nHeads / nKV;
    prm.scaleLog2 = invSqrt * kLog2e;
    if (kvHalf) return hd == 64 ? exact16<64>(prm, st) : exact16<128>(prm, st);
    if (hd == 64) return exact32<64>(prm, st);
    return hd == 128 ? exact32<128>(prm, st) : exact32<256>(prm, st);
}

}  // namespace tc
