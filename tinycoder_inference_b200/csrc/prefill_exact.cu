// prefill_exact.cu -- causal attention of several query rows in f32 arithmetic, over the f32 or fp16 store, without
// scratch: what a session without room for fp16 twins runs, and the launches whose position lives on the device.
//
// What it replaces: kWarpAttention / kWarpAttentionPos and kQ35WarpAttention of the reference
// (include/gpu/GpuAttentionKernels.hpp:211-272, 537-599; include/gpu/GpuQwen35Kernels.hpp:2437-2492): row s attends
// cache rows [0, pos + s], score = dot(q, k) * invSqrt, online softmax with exp2, out = sum p v / sum p.
//
// Over the f32 store every operand is an fp16 pair, x = 2^e (hi + lo) with a power of two per row, and a product is three on the
// tensor cores (mma.sync.m16n8k16: hi*hi + lo*hi + hi*lo, f32 accumulation): 22 bits of every factor like 3xTF32, at half the
// products and half the shared memory.  A row's scale is its own: K's goes into the score, V's into the probability.
//
// What bounds it: the issue slots.  With 8 query rows at a time (the causal form of the decode kernels, which stays for
// few rows behind a long prefix: prefillExactWins below) every warp takes K and V apart for itself.  Here a block of 32 query rows of
// one q head does that once per stage, into planes in shared memory: loader warps (loads, the rows' exponents, the pairs)
// fill one buffer while the computing warps, 16 rows x TG tokens each, work on the other.  Done by the
// computing warps between two barriers, as tf32 planes, a stage of 128 tokens at head_dim 64 took 3.9 us (1.6 of them products); with
// four loader warps and 9900 warp instructions in all 3.3, with eight and 8700 2.2 (half of the issue slots, a third of the
// tensor pipe).  The
// four token groups of a block take their share of every stage (a short prompt is a chain of stages, not a matter of
// bytes) and are put together at the end.  The late rows of all heads come first, so that what starts last is short.
// Measured, tf32 planes -> this: 512 rows of 14 / 2 / 64 17.7 -> 12.5 us, 512 behind 3000 200 -> 113; 512 rows of 28 / 4 / 128
// 59 -> 41, 512 behind 512 178 -> 116; 512 rows of 16 / 2 / 256 75 -> 46, 512 behind 512 215 -> 120.  fp16 store, 8-row form -> this: 100
// rows of 28 / 4 / 128 15.0 -> 6.4 us, 512 behind 512 107 -> 71, 2000 rows of 8 / 4 / 64 81 -> 40.
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
    static constexpr int kLoaders = HD > 128 ? 4 : 8, kThreads = (kExactWarps + kLoaders) * 32;
    static constexpr int kLd = HD + 8;  // halves per row of a plane: eight rows hit different banks
    static constexpr int kPlane = kStage * kLd;
    // halves: planes (hi, lo) of q [kRows][kLd], of K [NB][kStage][kLd], of V; then floats: scales of q's, K's and V's rows
    static constexpr int kQ = 0, kK = 2 * kRows * kLd, kV = kK + 2 * NB * kPlane, kHalves = kV + 2 * NB * kPlane;
    static constexpr int kScaleQ = 0, kScaleK = kRows, kScaleV = kScaleK + NB * kStage, kFloats = kScaleV + NB * kStage;
    static constexpr size_t kOperands = 2 * static_cast<size_t>(kHalves) + 4 * kFloats;
    static constexpr size_t kFold = 4 * static_cast<size_t>(kExactNH * kRows * (HD + 4));  // per group: O and (m, l) of every row
    static constexpr size_t kBytes = (kOperands > kFold ? kOperands : kFold) + 16;
    static_assert(kBytes <= 227 * 1024, "shared memory of an SM");
    static_assert(kHalves % 8 == 0, "16-byte accesses");
};

// two numbers as fp16 hi + lo pairs (22 significant bits)
__device__ __forceinline__ void splitPair(float a, float b, uint32_t &hi, uint32_t &lo) {
    hi = packHalf2(a, b);
    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
    const float2 r = __ffma2_rn(f, make_float2(-1.0f, -1.0f), make_float2(a, b));
    lo = packHalf2(r.x, r.y);
}
// Rows in powers of two: a row whose largest magnitude is in [2^e, 2^(e + 1)) is scaled into [2^14, 2^15), where the pairs keep 22 bits of
// every element down to 2^-17 of it, and 2^-39 of it of the smaller ones.  `x`: N pieces of such rows by the lanes of a warp; e gets
// the bits of 2^e of each (the rows that a warp holds at once share theirs).  Infinities and NaN stay out of it: they stay what they are
// in the planes, and leave the other elements their scale.
template <int N, int NV>
__device__ __forceinline__ void rowExponents(const float4 (&x)[N][NV], uint32_t (&e)[N]) {
    auto largest = [&](int i, auto of) {
        float m = 0.0f;
#pragma unroll
        for (int v = 0; v < NV; ++v) m = fmaxf(fmaxf(m, fmaxf(of(x[i][v].x), of(x[i][v].y))), fmaxf(of(x[i][v].z), of(x[i][v].w)));
        return __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    };
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = largest(i, [](float a) { return fabsf(a); }), top = max(top, e[i]);
    if (top >= 0x7f800000u) {  // warp-uniform
#pragma unroll
        for (int i = 0; i < N; ++i) e[i] = largest(i, [](float a) { return fabsf(a) < INFINITY ? fabsf(a) : 0.0f; });
    }
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = max(e[i] & 0x7f800000u, 15u << 23);
}
__device__ __forceinline__ float exactScale(uint32_t e) { return __uint_as_float((268u << 23) - e); }

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
    // hi and lo parts of a piece of a row, into row r of the planes at `plane` (`lo` halves apart)
    auto place = [&](__half *plane, uint32_t lo, const float4 (&x)[NV], float scale, uint32_t r) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            uint2 h, l;
            const float2 s2 = make_float2(scale, scale), a = __fmul2_rn(make_float2(x[v].x, x[v].y), s2), b = __fmul2_rn(make_float2(x[v].z, x[v].w), s2);
            splitPair(a.x, a.y, h.x, l.x);
            splitPair(b.x, b.y, h.y, l.y);
            __half *at = plane + r * LD + (unit + 32u * v) * 4u;
            *reinterpret_cast<uint2 *>(at) = h;
            *reinterpret_cast<uint2 *>(at + lo) = l;
        }
    };

    if (warp >= kExactWarps) {
        // (8 x 32 x 96 + 8 x 32 x 160 registers = the 512 x 128 of the launch)
        if constexpr (HD <= 128) asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
        // ---- loaders: rows of a stage through registers into the planes, K and V in turn, the next ones on their way meanwhile ----
        constexpr uint32_t LW = S::kLoaders, N = S::kStage / (LW * RW), H = HD > 128 ? 2 : 1, NH = N / H;  // units of a warp: H halves of NH
        static_assert(NH * H * LW * RW == S::kStage, "even shares");
        const uint32_t lw = warp - kExactWarps, kvHead = head / p.group;
        const size_t stride = static_cast<size_t>(p.nKV) * (HD / 4);
        const float4 *gk = static_cast<const float4 *>(p.k) + static_cast<size_t>(kvHead) * (HD / 4);
        const float4 *gv = static_cast<const float4 *>(p.v) + static_cast<size_t>(kvHead) * (HD / 4);
        auto rowOf = [&](uint32_t i) { return (i * LW + lw) * RW + sub; };
        // (rows behind the last one attended are zeros: 0 x NaN would be NaN)
        auto load = [&](float4 (&x)[NH][NV], const float4 *src, uint32_t st, uint32_t half) {
            const uint32_t tok0 = st * S::kStage + rowOf(half * NH);
            const float4 *at = src + tok0 * stride + unit;
            if ((st + 1u) * S::kStage <= len) {  // (a branch, not a condition per load)
#pragma unroll
                for (uint32_t i = 0; i < NH; ++i)
#pragma unroll
                    for (int v = 0; v < NV; ++v) x[i][v] = __ldg(at + i * (LW * RW * stride) + 32u * v);
                return;
            }
#pragma unroll
            for (uint32_t i = 0; i < NH; ++i)
#pragma unroll
                for (int v = 0; v < NV; ++v)
                    x[i][v] = tok0 + i * (LW * RW) < len ? __ldg(at + i * (LW * RW * stride) + 32u * v) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        auto put = [&](const float4 (&x)[NH][NV], __half *plane, float *scales, uint32_t half, bool isV) {
            uint32_t e[NH];
            rowExponents<NH, NV>(x, e);
#pragma unroll
            for (uint32_t i = 0; i < NH; ++i) {
                const uint32_t r = rowOf(half * NH + i);
                place(plane, S::kPlane, x[i], exactScale(e[i]), r);
                // V: 2^e, the probabilities carry it; K: what undoes the scale
                if (unit == 0) scales[r] = __uint_as_float(isV ? e[i] : e[i] - (14u << 23));
            }
        };
        float4 a[NH][NV], b[NH][NV];
        load(a, gk, 0, 0);
        load(b, H == 1 ? gv : gk, 0, H - 1);
        for (uint32_t st = 0; st < nStages; ++st) {
            const uint32_t buf = st % NB;
            __half *pk = sh + S::kK + buf * 2 * S::kPlane, *pv = sh + S::kV + buf * 2 * S::kPlane;
            float *sk = sf + S::kScaleK + buf * S::kStage, *sv = sf + S::kScaleV + buf * S::kStage;
            if (st >= NB) namedBarSync(kFreeK + buf, kAll);
            put(a, pk, sk, 0, false);
            if (H == 1) {
                if (st + 1 < nStages) load(a, gk, st + 1, 0);
                namedBarArrive(kFullK + buf, kAll);
                if (st >= NB) namedBarSync(kFreeV + buf, kAll);
                put(b, pv, sv, 0, true);
                if (st + 1 < nStages) load(b, gv, st + 1, 0);
                namedBarArrive(kFullV + buf, kAll);
            } else {
                load(a, gv, st, 0);
                put(b, pk, sk, 1, false);
                load(b, gv, st, 1);
                namedBarArrive(kFullK + buf, kAll);
                if (st >= NB) namedBarSync(kFreeV + buf, kAll);
                put(a, pv, sv, 0, true);
                if (st + 1 < nStages) load(a, gk, st + 1, 0);
                put(b, pv, sv, 1, true);
                if (st + 1 < nStages) load(b, gk, st + 1, 1);
                namedBarArrive(kFullV + buf, kAll);
            }
        }
        return;
    }

    if constexpr (HD <= 128) asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
    const uint32_t g = lane >> 2, t = lane & 3u, rt = warp % RT, nh = warp / RT;
    {   // q, the same way
        constexpr uint32_t N = S::kRows / (kExactWarps * RW);
        float4 x[N][NV];
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const uint32_t r = (i * kExactWarps + warp) * RW + sub;
#pragma unroll
            for (int v = 0; v < NV; ++v)
                x[i][v] = r < rows ? __ldg(reinterpret_cast<const float4 *>(p.q + (static_cast<size_t>(row0 + r) * p.nHeads + head) * HD) + unit + 32u * v)
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        uint32_t e[N];
        rowExponents<N, NV>(x, e);
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const uint32_t r = (i * kExactWarps + warp) * RW + sub;
            place(sh + S::kQ, S::kRows * LD, x[i], exactScale(e[i]), r);
            if (unit == 0) sf[S::kScaleQ + r] = p.scaleLog2 * __uint_as_float(e[i] - (14u << 23));
        }
    }
    namedBarSync(kFoldBar, kExactThreads);
    const float cs0 = sf[S::kScaleQ + rt * 16u + g], cs1 = sf[S::kScaleQ + rt * 16u + g + 8u];

    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    float m0 = kNegBig, m1 = kNegBig, l0 = 0.0f, l1 = 0.0f;
    // this thread's query rows (g and g + 8 of the warp's tile) see tokens below:
    const uint32_t lim0 = pos0 + row0 + rt * 16u + g + 1u, lim1 = lim0 + 8u;
    const uint32_t warpLimit = min(len, pos0 + row0 + rt * 16u + 16u);  // no row of the warp's tile sees further

    // ldmatrix: lane i delivers row i % 8 of 8x8 block i / 8
    const uint32_t aAddr = smemAddr(sh + S::kQ + (rt * 16u + (lane & 15u)) * LD + (lane >> 4) * 8u);
    // K: blocks (tokens 0-7, dims 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15)
    const uint32_t kAddr = smemAddr(sh + S::kK + (nh * TG + (lane & 7u) + (lane >> 4) * 8u) * LD + ((lane >> 3) & 1u) * 8u);
    // V, transposed: blocks (tokens 0-7, dims 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
    const uint32_t vAddr = smemAddr(sh + S::kV + (nh * TG + (lane & 15u)) * LD + (lane >> 4) * 8u);
    constexpr uint32_t kLoAt = S::kPlane * 2, kBufAt = 2 * kLoAt;  // bytes

    for (uint32_t st = 0; st < nStages; ++st) {
        const uint32_t buf = st % NB, tok0 = st * S::kStage + nh * TG;
        const bool active = tok0 < warpLimit, again = st + NB < nStages;  // (both warp-uniform)
        float s[NT][4], x[NT][4];  // hi*hi, and the cross terms
        namedBarSync(kFullK + buf, kAll);
        if (active) {
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
                    const uint32_t at = kAddr + buf * kBufAt + n * (16 * LD * 2) + ks * 32;
                    ldmatrixX4(bh[n][0], bh[n][1], bh[n][2], bh[n][3], at);
                    ldmatrixX4(bl[n][0], bl[n][1], bl[n][2], bl[n][3], at + kLoAt);
                }
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(s[n], ah[0], ah[1], ah[2], ah[3], bh[n / 2][n % 2 * 2], bh[n / 2][n % 2 * 2 + 1]);
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(x[n], al[0], al[1], al[2], al[3], bh[n / 2][n % 2 * 2], bh[n / 2][n % 2 * 2 + 1]);
#pragma unroll
                for (int n = 0; n < NT; ++n) mmaF16(x[n], ah[0], ah[1], ah[2], ah[3], bl[n / 2][n % 2 * 2], bl[n / 2][n % 2 * 2 + 1]);
            }
            // ---- online softmax: this thread has tokens 2t, 2t + 1 of every 8, rows g and g + 8 ----
            float mx0 = kNegBig, mx1 = kNegBig;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float2 sk = *reinterpret_cast<const float2 *>(sf + S::kScaleK + buf * S::kStage + nh * TG + 8 * n + 2 * t);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t tok = tok0 + 8 * n + 2 * t + i;
                    const float sc = i ? sk.y : sk.x;
                    s[n][i] = tok < lim0 ? (s[n][i] + x[n][i]) * (sc * cs0) : -INFINITY;
                    s[n][2 + i] = tok < lim1 ? (s[n][2 + i] + x[n][2 + i]) * (sc * cs1) : -INFINITY;
                    mx0 = fmaxf(mx0, s[n][i]);
                    mx1 = fmaxf(mx1, s[n][2 + i]);
                }
            }
            __syncwarp();  // (every lane has read its part of K and of its scales)
            if (again) namedBarArrive(kFreeK + buf, kAll);
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
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                s[n][0] = fastExp2(s[n][0] - m0), s[n][1] = fastExp2(s[n][1] - m0);
                s[n][2] = fastExp2(s[n][2] - m1), s[n][3] = fastExp2(s[n][3] - m1);
                l0 += s[n][0] + s[n][1];
                l1 += s[n][2] + s[n][3];
            }
        } else if (again) {
            namedBarArrive(kFreeK + buf, kAll);
        }
        namedBarSync(kFullV + buf, kAll);
        if (active) {
            // ---- O += P V, 16 tokens at a time: the accumulator layout of the scores is the A operand's.  The probabilities take the
            // scales of V's rows along, and every query row a power of two of its own, out of its largest product: with one for the group a
            // row of V that is masked, or weighs nothing, pushed the probabilities of the others out of the pairs' range ----
            const float *sv = sf + S::kScaleV + buf * S::kStage + nh * TG;
            float top0 = 0.0f, top1 = 0.0f;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float2 w = *reinterpret_cast<const float2 *>(sv + 8 * n + 2 * t);
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] *= i & 1 ? w.y : w.x;
                top0 = fmaxf(top0, fmaxf(s[n][0], s[n][1]));
                top1 = fmaxf(top1, fmaxf(s[n][2], s[n][3]));
            }
#pragma unroll
            for (int off = 1; off <= 2; off <<= 1) {
                top0 = fmaxf(top0, __shfl_xor_sync(0xffffffffu, top0, off));
                top1 = fmaxf(top1, __shfl_xor_sync(0xffffffffu, top1, off));
            }
            const uint32_t e0 = max(__float_as_uint(top0) & 0x7f800000u, 15u << 23), e1 = max(__float_as_uint(top1) & 0x7f800000u, 15u << 23);
            const float in0 = exactScale(e0), in1 = exactScale(e1);
            uint32_t ph[NT / 2][4], pl[NT / 2][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                splitPair(s[n][0] * in0, s[n][1] * in0, ph[n / 2][n % 2 * 2], pl[n / 2][n % 2 * 2]);
                splitPair(s[n][2] * in1, s[n][3] * in1, ph[n / 2][n % 2 * 2 + 1], pl[n / 2][n % 2 * 2 + 1]);
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
                        const uint32_t at = vAddr + buf * kBufAt + n * (16 * LD * 2) + (d0 + d) * 32;
                        ldmatrixX4Trans(bh[d][0], bh[d][1], bh[d][2], bh[d][3], at);
                        ldmatrixX4Trans(bl[d][0], bl[d][1], bl[d][2], bl[d][3], at + kLoAt);
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
                    for (int i = 0; i < 4; ++i) o[2 * d0 + d][i] = fmaf(sum[d][i] + cross[d][i], i & 2 ? out1 : out0, o[2 * d0 + d][i]);
            }
            __syncwarp();
        }
        if (again) namedBarArrive(kFreeV + buf, kAll);
    }
    exactFold<HD>(sm, o, m0, m1, l0, l1, nh, rt, rows, p.out + (static_cast<size_t>(row0) * p.nHeads + head) * HD,
                  static_cast<size_t>(p.nHeads) * HD);
}

// ---- fp16 store ------------------------------------------------------------------------------------------
// fp16 K and V are operands as they are (m16n8k16, twice the rate of the tf32 products and no third one); q, normalised by
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
    static constexpr ExactCost k32[3] = {{3.0f, 0.0103f, 3.4f, 0.0164f}, {4.2f, 0.0193f, 3.4f, 0.0365f}, {5.1f, 0.0548f, 6.0f, 0.0727f}};
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
