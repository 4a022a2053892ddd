// prefill_exact.cu -- causal attention of several query rows in f32 arithmetic, over the f32 or fp16 store, without
// scratch: what a session without room for fp16 twins runs, and the launches whose position lives on the device.
//
// What it replaces: kWarpAttention / kWarpAttentionPos and kQ35WarpAttention of the reference
// (include/gpu/GpuAttentionKernels.hpp:211-272, 537-599; include/gpu/GpuQwen35Kernels.hpp:2437-2492): row s attends
// cache rows [0, pos + s], score = dot(q, k) * invSqrt, online softmax with exp2, out = sum p v / sum p.
//
// Over the f32 store the products run as 3xTF32 on the tensor cores (mma.sync.m16n8k8: x = hi + lo, both tf32; hi*hi +
// lo*hi + hi*lo keeps about 21 mantissa bits and the full exponent range, f32 accumulation).
//
// What bounds it: the issue slots.  With 8 query rows at a time (the causal form of the decode kernels, which stays for
// few rows behind a long prefix: prefillExactWins below) every warp splits K and V into hi and lo for itself, half of the 370
// instructions it spends on a 16-token tile.  Here a block of 32 query rows of one q head splits a stage of K and V once
// into planes in shared memory, and a warp works on 16 rows x TG tokens: ldmatrix operands, three products each.  The
// four token groups of a block take their share of every stage (a short prompt is a chain of stages, not a matter of
// bytes) and are put together at the end.  (Blocks of 64 rows and two token groups leave fewer and longer chains: 512
// rows of 28 / 4 / 128 83 us against 79.)  The late rows of all heads come first, so that what starts last is short: that
// form head by head took 79 us, 62 now (fp16, 512 behind 512 of 28 / 4 / 128, is the one that lost: 67.6 -> 70.7).  Measured (8-row form -> this one): f32 512 rows of 14 / 2 / 64 39.7 -> 18.7 us,
// of 28 / 4 / 128 120 -> 62, 333 of 16 / 2 / 256 77 -> 52; fp16 100 rows of 28 / 4 / 128 15.0 -> 6.4 us, 512 behind 512
// 107 -> 71, 2000 rows of 8 / 4 / 64 81 -> 40.
//
// What keeps it exact: a tensor-core product drops the bits of a running sum that do not fit, and those losses add up
// along a chain.  The 8-row form has up to sixteen warps and so as many sums per output; four token groups with one
// running sum each were further from a 64-bit evaluation (head_dim 64, 200 rows behind 6000: f32 5.6e-6 -> 1.1e-5 of the
// result's norm, fp16 512 behind 1000 5.5e-7 -> 9.1e-7).  So where it is needed (kOwnSums, and the fp16 form) a stage's
// products are summed by themselves, the small terms apart (f32) or first (fp16), and added to O in f32: 4.0e-7 and 2.9e-7,
// for 1 - 3 % more time.  At head_dim 128 and 256 the f32 form's short stages are no further off than the 8-row form was, and keep one sum.
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

// RT 16-row tiles of query rows x NH token groups = warps of a block.
static constexpr int kExactRT = 2, kExactNH = 4, kExactWarps = kExactRT * kExactNH, kExactRows = 16 * kExactRT;

// TG tokens of a stage per group: what shared memory (head_dim 256) and registers carry.
template <int HD>
struct ExactShape {
    static constexpr int TG = 2048 / HD, kRows = kExactRows, kStage = kExactNH * TG;
    static constexpr bool kOwnSums = HD == 64;  // see the head of the file
    static constexpr int kLd = HD + 4;  // floats per row of a plane: eight rows hit different banks
    static constexpr int kQ = 0;                                  // planes (hi, lo): q [kRows][kLd],
    static constexpr int kK = kQ + 2 * kRows * kLd;               // K [kStage][kLd],
    // V [kStage][kLd]
    static constexpr int kV = kK + 2 * kStage * kLd;
    static constexpr int kFloats = kV + 2 * kStage * kLd;
    static constexpr int kFold = kExactNH * kRows * (HD + 4);           // per group: O and (m, l) of every row
    static constexpr size_t kBytes = 4 * static_cast<size_t>(kFloats > kFold ? kFloats : kFold) + 16;
    static_assert(kBytes <= 227 * 1024, "shared memory of an SM");
};

__device__ __forceinline__ void splitTf32(float x, float &hi, float &lo) {
    hi = __uint_as_float(toTf32(x));
    lo = __uint_as_float(toTf32(x - hi));
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
    __syncthreads();  // the operands are done with: the fold's scratch takes their place
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
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < rows * (HD / 4); i += kExactWarps * 32) {
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
__global__ void __launch_bounds__(kExactWarps * 32, 1) prefillExactKernel(const __grid_constant__ PrefillExactParams p) {
    using S = ExactShape<HD>;
    constexpr int RT = kExactRT, TG = S::TG, LD = S::kLd, NT = TG / 8;
    constexpr uint32_t kThreads = kExactWarps * 32;
    extern __shared__ __align__(16) float sm[];
    float *sQ = sm + S::kQ, *sK = sm + S::kK, *sV = sm + S::kV;
    gridDepWait();
    gridDepLaunch();

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t rt = warp % RT, nh = warp / RT;
    const uint32_t blk = gridDim.y - 1u - blockIdx.y, head = blockIdx.x;  // late rows (long prefixes) of all heads first
    const uint32_t row0 = blk * S::kRows, rows = min(static_cast<uint32_t>(S::kRows), p.qRows - row0);
    const uint32_t pos0 = p.devPos ? p.devPos[0] : p.cachePos;
    const uint64_t wanted = static_cast<uint64_t>(pos0) + row0 + rows;
    const uint32_t len = static_cast<uint32_t>(wanted < p.totalRows ? wanted : p.totalRows);  // (a device position past the store)
    const uint32_t kvHead = head / p.group;

    // (the loads of q first, those of the first stage behind them, then q's planes: one wait for both)
    constexpr uint32_t kQUnits = S::kRows * (HD / 4), kQPer = kQUnits / kThreads;
    static_assert(kQUnits % kThreads == 0, "even shares");
    float4 qv[kQPer];
#pragma unroll
    for (uint32_t i = 0; i < kQPer; ++i) {
        const uint32_t idx = threadIdx.x + i * kThreads, r = idx / (HD / 4), c = (idx % (HD / 4)) * 4;
        qv[i] = r < rows ? __ldg(reinterpret_cast<const float4 *>(p.q + (static_cast<size_t>(row0 + r) * p.nHeads + head) * HD + c))
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    }

    // A stage's rows pass through registers: requested while the stage before it is worked on, split into the planes
    // when that is done.  Rows behind the last one attended are zeros (0 x NaN would be NaN).
    constexpr uint32_t kUnits = S::kStage * (HD / 4), kPer = kUnits / kThreads;  // 4-element units, per thread
    static_assert(kUnits % kThreads == 0, "even shares");
    float4 uk[kPer], uv[kPer];
    const size_t stride = static_cast<size_t>(p.nKV) * (HD / 4);
    const float4 *gk = static_cast<const float4 *>(p.k) + static_cast<size_t>(kvHead) * (HD / 4);
    const float4 *gv = static_cast<const float4 *>(p.v) + static_cast<size_t>(kvHead) * (HD / 4);
    auto request = [&](uint32_t tok0) {
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            const uint32_t idx = threadIdx.x + i * kThreads, r = idx / (HD / 4), c = idx % (HD / 4);
            uk[i] = make_float4(0.f, 0.f, 0.f, 0.f), uv[i] = uk[i];
            if (tok0 + r < len) {
                uk[i] = __ldg(gk + (tok0 + r) * stride + c);
                uv[i] = __ldg(gv + (tok0 + r) * stride + c);
            }
        }
    };
    auto place = [&](float *plane, const float4 &u, uint32_t r, uint32_t c) {
        float4 h, l;
        splitTf32(u.x, h.x, l.x);
        splitTf32(u.y, h.y, l.y);
        splitTf32(u.z, h.z, l.z);
        splitTf32(u.w, h.w, l.w);
        *reinterpret_cast<float4 *>(plane + r * LD + c) = h;
        *reinterpret_cast<float4 *>(plane + (S::kStage + r) * LD + c) = l;
    };

    request(0);
    // q: hi and lo planes
#pragma unroll
    for (uint32_t i = 0; i < kQPer; ++i) {
        const uint32_t idx = threadIdx.x + i * kThreads, r = idx / (HD / 4), c = (idx % (HD / 4)) * 4;
        float4 h, l;
        splitTf32(qv[i].x, h.x, l.x);
        splitTf32(qv[i].y, h.y, l.y);
        splitTf32(qv[i].z, h.z, l.z);
        splitTf32(qv[i].w, h.w, l.w);
        *reinterpret_cast<float4 *>(sQ + r * LD + c) = h;
        *reinterpret_cast<float4 *>(sQ + (S::kRows + r) * LD + c) = l;
    }

    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    float m0 = kNegBig, m1 = kNegBig, l0 = 0.0f, l1 = 0.0f;
    // this thread's query rows (g and g + 8 of the warp's tile) see tokens below:
    const uint32_t lim0 = pos0 + row0 + rt * 16u + g + 1u, lim1 = lim0 + 8u;
    const uint32_t warpLimit = min(len, pos0 + row0 + rt * 16u + 16u);  // no row of the warp's tile sees further

    // ldmatrix addresses: lane i delivers row i % 8 of 8x4 block i / 8 (16 bytes of a plane row)
    const uint32_t aAddr = smemAddr(sQ + (rt * 16u + (lane & 7u) + ((lane >> 3) & 1u) * 8u) * LD + (lane >> 4) * 4u);
    // K operand: blocks (k 0-3, k 4-7) of the hi plane, then of the lo plane
    const uint32_t bRow = nh * TG + (lane & 7u) + (lane >> 4) * S::kStage;
    const uint32_t bAddr = smemAddr(sK + bRow * LD + ((lane >> 3) & 1u) * 4u);

    const uint32_t nStages = (len + S::kStage - 1) / S::kStage;
    for (uint32_t st = 0; st < nStages; ++st) {
        __syncthreads();  // the planes are free (and, the first time, q's are complete)
#pragma unroll
        for (uint32_t i = 0; i < kPer; ++i) {
            const uint32_t idx = threadIdx.x + i * kThreads, r = idx / (HD / 4), c = idx % (HD / 4) * 4;
            place(sK, uk[i], r, c);
            place(sV, uv[i], r, c);
        }
        __syncthreads();
        if (st + 1 < nStages) request((st + 1) * S::kStage);
        const uint32_t tok0 = st * S::kStage + nh * TG;
        if (tok0 >= warpLimit) continue;  // warp-uniform

        // ---- scores: 16 rows x TG tokens ----
        float s[NT][4], x[NT][4], y[NT][4];  // hi*hi, and the cross terms
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[n][i] = x[n][i] = y[n][i] = 0.0f;
#pragma unroll 2
        for (int ks = 0; ks < HD / 8; ++ks) {
            uint32_t ah[4], al[4];
            ldmatrixX4(ah[0], ah[1], ah[2], ah[3], aAddr + ks * 32);
            ldmatrixX4(al[0], al[1], al[2], al[3], aAddr + (S::kRows * LD) * 4 + ks * 32);
            // (no product waits for the one in front of it: the chains of the NT token tiles and of the cross terms alternate)
            uint32_t b[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) ldmatrixX4(b[n][0], b[n][1], b[n][2], b[n][3], bAddr + n * (8 * LD * 4) + ks * 32);
#pragma unroll
            for (int n = 0; n < NT; ++n) mmaTf32(s[n], ah[0], ah[1], ah[2], ah[3], b[n][0], b[n][1]);
#pragma unroll
            for (int n = 0; n < NT; ++n) mmaTf32(x[n], al[0], al[1], al[2], al[3], b[n][0], b[n][1]);
#pragma unroll
            for (int n = 0; n < NT; ++n) mmaTf32(y[n], ah[0], ah[1], ah[2], ah[3], b[n][2], b[n][3]);
        }
        // ---- online softmax: this thread has tokens 2t, 2t + 1 of every 8, rows g and g + 8 ----
        float mx0 = kNegBig, mx1 = kNegBig;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t tok = tok0 + 8 * n + 2 * t + i;
                s[n][i] = tok < lim0 ? (s[n][i] + (x[n][i] + y[n][i])) * p.scaleLog2 : -INFINITY;
                s[n][2 + i] = tok < lim1 ? (s[n][2 + i] + (x[n][2 + i] + y[n][2 + i])) * p.scaleLog2 : -INFINITY;
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
        // ---- O += P V.  The k slots t / t + 4 of an 8-token step stand for tokens 2t / 2t + 1: the accumulator layout
        // of the scores is the A operand then, and V is read with rows 2t, 2t + 1 ----
        float own[S::kOwnSums ? HD / 8 : 1][4], ownCross[S::kOwnSums ? HD / 8 : 1][4];  // this stage's hi*hi, and the cross terms
        auto sum = [&](int d) -> float (&)[4] { return S::kOwnSums ? own[S::kOwnSums ? d : 0] : o[d]; };
        auto cross = [&](int d) -> float (&)[4] { return S::kOwnSums ? ownCross[S::kOwnSums ? d : 0] : o[d]; };
        if (S::kOwnSums) {
#pragma unroll
            for (int d = 0; d < HD / 8; ++d)
#pragma unroll
                for (int i = 0; i < 4; ++i) sum(d)[i] = cross(d)[i] = 0.0f;
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float ph[4], pl[4];
            {
                const float p0 = fastExp2(s[n][0] - m0), p1 = fastExp2(s[n][1] - m0);
                const float p2 = fastExp2(s[n][2] - m1), p3 = fastExp2(s[n][3] - m1);
                l0 += p0 + p1;
                l1 += p2 + p3;
                splitTf32(p0, ph[0], pl[0]);
                splitTf32(p2, ph[1], pl[1]);
                splitTf32(p1, ph[2], pl[2]);
                splitTf32(p3, ph[3], pl[3]);
            }
            auto u = [](float f) { return __float_as_uint(f); };
            const float *v0 = sV + (nh * TG + 8 * n + 2 * t) * LD + g, *v1 = v0 + LD;
            constexpr int DB = 4;  // dim tiles at a time, their chains alternating
#pragma unroll
            for (int d0 = 0; d0 < HD / 8; d0 += DB) {
                uint32_t b[DB][4];
#pragma unroll
                for (int d = 0; d < DB; ++d) {
                    const float *a0 = v0 + 8 * (d0 + d), *a1 = v1 + 8 * (d0 + d);
                    b[d][0] = u(a0[0]), b[d][1] = u(a1[0]);
                    b[d][2] = u(a0[S::kStage * LD]), b[d][3] = u(a1[S::kStage * LD]);
                }
#pragma unroll
                for (int d = 0; d < DB; ++d) mmaTf32(sum(d0 + d), u(ph[0]), u(ph[1]), u(ph[2]), u(ph[3]), b[d][0], b[d][1]);
#pragma unroll
                for (int d = 0; d < DB; ++d) mmaTf32(cross(d0 + d), u(pl[0]), u(pl[1]), u(pl[2]), u(pl[3]), b[d][0], b[d][1]);
#pragma unroll
                for (int d = 0; d < DB; ++d) mmaTf32(cross(d0 + d), u(ph[0]), u(ph[1]), u(ph[2]), u(ph[3]), b[d][2], b[d][3]);
            }
        }
        if (S::kOwnSums) {
#pragma unroll
            for (int d = 0; d < HD / 8; ++d)
#pragma unroll
                for (int i = 0; i < 4; ++i) o[d][i] += sum(d)[i] + cross(d)[i];
        }
    }
    exactFold<HD>(sm, o, m0, m1, l0, l1, nh, rt, rows,
                                                p.out + (static_cast<size_t>(row0) * p.nHeads + head) * HD,
                                                static_cast<size_t>(p.nHeads) * HD);
}

// ---- fp16 store ------------------------------------------------------------------------------------------
// fp16 K and V are operands as they are (m16n8k16, twice the rate of the tf32 products and no third one); q, normalised by
// a power of two per row, and the probabilities are fp16 hi + lo pairs (two products, ~22 mantissa bits), as in
// decode_kv16.cu.  Stages come in by cp.async, two deep.
template <int HD>
struct ExactHalfShape {
    static constexpr int TG = 32, BPS = HD == 64 ? 2 : 1, kRows = kExactRows, kStage = kExactNH * TG;
    static constexpr int kLd = HD + 8;                       // halves per row: eight rows hit different banks
    static constexpr int kQ = 0;                             // q hi, lo [kRows][kLd]
    static constexpr int kKV = 2 * kRows * kLd;              // [2 stages][K, V][kStage][kLd]
    static constexpr int kHalves = kKV + 4 * kStage * kLd;
    static constexpr int kFold = 2 * kExactNH * kRows * (HD + 4);  // in halves
    static constexpr size_t kBytes = 2 * static_cast<size_t>(kHalves > kFold ? kHalves : kFold) + 16;
    static_assert(kBytes * BPS <= 227 * 1024, "shared memory of an SM");
};

template <int HD>
__global__ void __launch_bounds__(kExactWarps * 32, ExactHalfShape<HD>::BPS)
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
    return launchDependent(kern, dim3(prm.nHeads, (prm.qRows + kExactRows - 1) / kExactRows), kExactWarps * 32, S::kBytes, st, 1,
                           prm);
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
    static constexpr ExactCost k32[3] = {{3.0f, 0.0103f, 3.5f, 0.0296f}, {4.2f, 0.0193f, 4.0f, 0.0595f}, {5.1f, 0.0548f, 5.6f, 0.13f}};
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
