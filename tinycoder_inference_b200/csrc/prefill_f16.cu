// prefill_f16.cu -- causal prefill attention on tcgen05 tensor cores (fp16 operands,
// f32 accumulation in TMEM).
//
// What it replaces: the reference's materialised dense prefill -- kF32ToF16 twins of
// q and of the stored K/V rows, one cuBLAS GEMM per q head for QK^T (f32 scores of
// seqLen^2 per head), kAttnSoftmaxCausal, one cuBLAS GEMM per q head for PV
// (src/cpp/core/cuda/forward/GPUComputeForward.cu:3937-4026;
// include/gpu/GpuAttentionKernels.hpp:323-353).  Same arithmetic contract: fp16
// products, f32 accumulation, f32 softmax with exp2 and the scale applied to the
// scores, probabilities rounded to fp16 -- but flash-style, so the score matrix
// never exists and the sequence length is not capped at 512.
//
// One persistent block per SM walks work items: a q head x 256 query rows = two 128-row query
// tiles A and B, KV tiles of 64 tokens.  A call with fewer such items than SMs takes items of ONE query
// tile whose KV tiles the two halves of the block share (even / odd) and put together at the end: 512 rows
// behind 3584 of 28 q heads of 128 take 48.6 us, with one half idle 55.5.  At head_dim 256 a block
// holds one query tile (2000 rows of 16 heads: 55.9 us, with 32-token KV tiles 79.0).
// Calls of so few one-tile items that blocks would be left without give each item to a cluster of 2 - 8 blocks, which share its KV
// tiles and put their results together through distributed shared memory (SHARED below).
// The first item of a block is its index, the following ones come from a
// counter, heavy (late) query blocks first; the mbarriers are initialised once, every ring index
// counts on from item to item, so the next item's loads and first score products run under the
// current item's epilogue.  Warp roles:
//   warps 0-3 / 4-7  softmax of tile A / B: thread r owns query row r, reads its scores of a KV
//              tile from TMEM (tcgen05.ld), keeps (m, l), writes the fp16 probabilities over the
//              first columns of the same S buffer (tcgen05.st) as the A operand of the PV product,
//              rescales O in TMEM only when the row maximum ran ahead by 2^8 (lazy rescale);
//              packed f32x2 arithmetic; normalises and stores the output rows (32-byte stores);
//   warp 8     TMA producer and scheduler: the query tiles per item, then K two tiles ahead of V
//              into rings of their own (cp.async.bulk.tensor, 128-byte swizzle = the canonical UMMA
//              shared-memory layout, so no register pass touches the operands); draws the next
//              item late in the current;
//   warps 9, 10  issue the score products of tile A / B: S_X(t) = Q_X K^T (M128 N64 K16 per
//              instruction), tcgen05.commit onto the softmax warps' barrier;
//   warps 11, 12  issue the P.V products of tile A / B: O_X += P_X(t) V (A from TMEM, B = V
//              MN-major from shared memory).  One elected thread of each issues (tc_tcgen05.cuh).
// S is DOUBLE-BUFFERED per query tile (head_dim 256: kAhead below): S_X(t+2) goes into the buffer P_X(t) leaves once its P.V
// product is complete, so S_X(t+1) is there when the softmax of tile t finishes.  TMEM (512
// columns): O_A, O_B (128 each, f32; one O of 256 at head_dim 256), S_{A,0}, S_{A,1}, S_{B,0},
// S_{B,1} (64 each).  Causality: a query tile only visits KV tiles up to its diagonal, the last
// two or three are masked element-wise; the query rows may sit behind an existing cache.
// In front of the kernel one launch (prefillRowsKernel) makes the fp16 twins of q, K and V and puts the
// call's new rows into the store; the attention kernel is its programmatic dependent.
// Every wait is bounded; a wait that runs out records an error bit, every other wait of the launch
// then gives up at once, the block frees its TMEM and returns.
#include <algorithm>
#include <cstring>

#include "decode_cluster.cuh"
#include "prefill_rows.cuh"
#include "tc_tcgen05.cuh"

namespace tc {

constexpr int kPfBM = 128;    // query rows per tile (two tiles per CTA)
constexpr int kPfBN = 64;     // tokens per KV tile
constexpr float kPfLazyLog2 = 8.0f;

// Everything between a call's f32 rows and the attention launch, in ONE launch: q to fp16 (the reference's kF32ToF16,
// GpuElementwiseKernels.hpp:92-101; GPUComputeForward.cu:3957-3968), rotated in place first in the dense models; the new
// K/V rows -- if the call brings them -- rotated and stored into the f32 / fp16 / int8 store (the arithmetic of
// kvAppendKernel and kvQuantKernel, bit for bit); the fp16 twins of all rows the call attends over (an fp16 store needs
// none: its layout is the twins'); and the int8 pool rows of the new positions beside an f32 store.  q goes four
// rotation pairs per thread; a K/V row of one kv head goes to a warp, lane i holding dims 4 i .. 4 i + 3 (and 128
// further on at head_dim 256), so its maximum is a shuffle away.
// HBM-bound for prompts: 4096 rows of 28 q / 4 kv heads of 128 with the mirror move 134 MB in 23.6 us, 5.7 TB/s (append and
// twins as launches of their own: 33 us, and the rows went through HBM twice); launch-bound for short ones.
struct PrefillRowsParams {
    float *q;              // [seqLen][nHeads][hd]; written back only when it is rotated
    uint2 *q16, *k16, *v16;
    PrefillKvStore st;
    PrefillNewRows nr;
    PrefillMirror mir;
    uint32_t seqLen, cachePos, nHeads, nKV;
    uint32_t qBlocks;      // APART: the first blocks, which work on q
    uint32_t prefetchBlocks;  // how many blocks pull the launch's inputs into L2 ahead of the wait
    unsigned int *err, *workCounter;
};

// What the launch reads, towards L2 while the one in front of it drains (the attention launch of the layer before leaves SMs idle
// one by one, and HBM all the while): 1 / prefetchBlocks of everything by each of the blocks that are resident first.  1900 rows
// in calls of 512 of 28 / 4 / 128, int8, two layers: 177.6 -> 172.4 us.
template <int HD>
__device__ __forceinline__ void prefetchRowsInputs(const PrefillRowsParams &p) {
    if (blockIdx.x >= p.prefetchBlocks || threadIdx.x >= 32u) return;
    auto pull = [&](const void *base, size_t bytes) {
        constexpr size_t kPiece = 4096;
        const size_t pieces = (bytes + kPiece - 1) / kPiece;
        for (size_t i = blockIdx.x + static_cast<size_t>(threadIdx.x) * p.prefetchBlocks; i < pieces; i += 32u * p.prefetchBlocks)
            prefetchBulkL2(static_cast<const uint8_t *>(base) + i * kPiece, static_cast<uint32_t>(min(kPiece, bytes - i * kPiece)));
    };
    const size_t row = static_cast<size_t>(p.nKV) * HD;
    pull(p.q, static_cast<size_t>(p.seqLen) * p.nHeads * HD * 4);
    if (p.nr.k != nullptr) pull(p.nr.k, p.seqLen * row * 4), pull(p.nr.v, p.seqLen * row * 4);
    if (p.k16 != nullptr) {
        const size_t have = (static_cast<size_t>(p.cachePos) + (p.nr.k != nullptr ? 0u : p.seqLen)) * row * (p.st.kind == 2 ? 1 : 4);
        pull(p.st.k, have), pull(p.st.v, have);
    }
}

// APART: the first qBlocks blocks work on q, the others on K and V; else every block does both, one after the other.
template <int HD, bool APART>
__global__ void __launch_bounds__(256) prefillRowsKernel(const __grid_constant__ PrefillRowsParams p) {
    prefetchRowsInputs<HD>(p);
    gridDepWait();
    gridDepLaunch();  // the attention launch may set itself up while this one drains (it waits before it lets anything else in)
    // the attention launch that follows in the stream hands out its work items through this counter
    if (blockIdx.x == 0 && threadIdx.x == 0) *p.workCounter = 0u;
    const bool forQ = !APART || blockIdx.x < p.qBlocks;
    const size_t tid = static_cast<size_t>(forQ ? blockIdx.x : blockIdx.x - p.qBlocks) * blockDim.x + threadIdx.x;
    const size_t stride = static_cast<size_t>(!APART ? gridDim.x : forQ ? p.qBlocks : gridDim.x - p.qBlocks) * blockDim.x;
    constexpr uint32_t half = HD / 2, perRow = half / 4, nvec = HD / 4;
    constexpr int MAXV = HD > 128 ? 2 : 1;  // float4 per lane and K/V row
    auto half4 = [](const float4 &x) { return make_uint2(packHalf2(x.x, x.y), packHalf2(x.z, x.w)); };
    auto rotate = [](float4 &a, float4 &b, const float4 &c, const float4 &s) {
        auto rot = [](float &x0, float &x1, float cc, float ss) {
            const float y = fmaf(x0, cc, -__fmul_rn(x1, ss));
            x1 = fmaf(x0, ss, __fmul_rn(x1, cc));
            x0 = y;
        };
        rot(a.x, b.x, c.x, s.x);
        rot(a.y, b.y, c.y, s.y);
        rot(a.z, b.z, c.z, s.z);
        rot(a.w, b.w, c.w, s.w);
    };
    const size_t qUnits = forQ ? static_cast<size_t>(p.seqLen) * p.nHeads * perRow : 0;
    constexpr int N = 4;  // units of a thread in flight
    for (size_t i0 = tid; i0 < qUnits; i0 += N * stride) {
        float4 x[N], y[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const size_t i = i0 + u * stride;
            if (i >= qUnits) continue;
            const float4 *a = reinterpret_cast<const float4 *>(p.q) + i / perRow * nvec + i % perRow;
            x[u] = a[0];
            y[u] = a[perRow];
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const size_t i = i0 + u * stride;
            if (i >= qUnits) continue;
            const size_t row = i / perRow, at = row * nvec + i % perRow;
            if (p.nr.cosT != nullptr) {
                const size_t t = (static_cast<size_t>(p.cachePos) + row / p.nHeads) * perRow + i % perRow;
                rotate(x[u], y[u], __ldg(reinterpret_cast<const float4 *>(p.nr.cosT) + t),
                       __ldg(reinterpret_cast<const float4 *>(p.nr.sinT) + t));
                reinterpret_cast<float4 *>(p.q)[at] = x[u];
                reinterpret_cast<float4 *>(p.q)[at + perRow] = y[u];
            }
            p.q16[at] = half4(x[u]);
            p.q16[at + perRow] = half4(y[u]);
        }
    }
    if (APART && forQ) return;
    const uint32_t lane = threadIdx.x & 31u;
    const size_t newFrom = static_cast<size_t>(p.cachePos) * p.nKV;            // first (row, kv head) of the call's rows
    const size_t end = newFrom + static_cast<size_t>(p.seqLen) * p.nKV;
    const bool bring = p.nr.k != nullptr;
    // (an fp16 store has nothing to do for rows that it already holds)
    const size_t begin = p.k16 != nullptr ? 0 : (bring ? newFrom : end);
    for (size_t rh = begin + (tid >> 5); rh < end; rh += stride >> 5) {
        const bool fresh = bring && rh >= newFrom;
        float4 kx[MAXV], vx[MAXV];
        bool active[MAXV];
#pragma unroll
        for (int u = 0; u < MAXV; ++u) {
            const uint32_t i4 = lane + 32u * u;
            active[u] = i4 < nvec;
            kx[u] = make_float4(0.f, 0.f, 0.f, 0.f), vx[u] = kx[u];
            if (!active[u]) continue;
            if (fresh) {
                kx[u] = __ldg(reinterpret_cast<const float4 *>(p.nr.k) + (rh - newFrom) * nvec + i4);
                vx[u] = __ldg(reinterpret_cast<const float4 *>(p.nr.v) + (rh - newFrom) * nvec + i4);
            } else if (p.st.kind == 2) {
                const uint32_t kb = __ldg(static_cast<const uint32_t *>(p.st.k) + rh * nvec + i4),
                               vb = __ldg(static_cast<const uint32_t *>(p.st.v) + rh * nvec + i4);
                const float sk = __ldg(p.st.ks + rh), sv = __ldg(p.st.vs + rh);
                auto b = [](uint32_t w, int i) { return static_cast<float>(static_cast<int8_t>((w >> (8 * i)) & 0xffu)); };
                kx[u] = make_float4(b(kb, 0) * sk, b(kb, 1) * sk, b(kb, 2) * sk, b(kb, 3) * sk);
                vx[u] = make_float4(b(vb, 0) * sv, b(vb, 1) * sv, b(vb, 2) * sv, b(vb, 3) * sv);
            } else {
                kx[u] = __ldg(static_cast<const float4 *>(p.st.k) + rh * nvec + i4);
                vx[u] = __ldg(static_cast<const float4 *>(p.st.v) + rh * nvec + i4);
            }
        }
        if (fresh && p.nr.cosT != nullptr) {  // warp-uniform
            const size_t at = static_cast<size_t>(rh / p.nKV) * half;
            if (MAXV > 1) {
                // the partner of a lane's first float4 is its second one
                rotate(kx[0], kx[MAXV - 1], __ldg(reinterpret_cast<const float4 *>(p.nr.cosT + at) + lane),
                       __ldg(reinterpret_cast<const float4 *>(p.nr.sinT + at) + lane));
            } else {
                // perRow lanes apart
                const bool low = lane < perRow;
                const uint32_t j = low ? lane : lane - perRow;
                float4 o;
                o.x = __shfl_xor_sync(0xffffffffu, kx[0].x, perRow);
                o.y = __shfl_xor_sync(0xffffffffu, kx[0].y, perRow);
                o.z = __shfl_xor_sync(0xffffffffu, kx[0].z, perRow);
                o.w = __shfl_xor_sync(0xffffffffu, kx[0].w, perRow);
                if (active[0]) {
                    float4 a = low ? kx[0] : o, b = low ? o : kx[0];
                    rotate(a, b, __ldg(reinterpret_cast<const float4 *>(p.nr.cosT + at) + j),
                           __ldg(reinterpret_cast<const float4 *>(p.nr.sinT + at) + j));
                    kx[0] = low ? a : b;
                }
            }
        }
        // int8 rows: of the store itself, or of the pool beside an f32 store
        const bool toStore8 = fresh && p.st.kind == 2;
        const bool toMirror = p.mir.k8 != nullptr && rh >= newFrom;
        if (toStore8 || toMirror) {  // warp-uniform
            auto amax4 = [](const float4 &x) { return fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))); };
            float mk = amax4(kx[0]), mv = amax4(vx[0]);
            if (MAXV > 1) mk = fmaxf(mk, amax4(kx[MAXV - 1])), mv = fmaxf(mv, amax4(vx[MAXV - 1]));
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                mk = fmaxf(mk, __shfl_xor_sync(0xffffffffu, mk, o));
                mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
            }
            const float sk = mk > 0.0f ? __fdiv_rn(mk, 127.0f) : 1.0f;
            const float sv = mv > 0.0f ? __fdiv_rn(mv, 127.0f) : 1.0f;
            const size_t dst = toStore8 ? rh : static_cast<size_t>(p.mir.dstRow) * p.nKV + (rh - newFrom);
            uint32_t *k8 = toStore8 ? static_cast<uint32_t *>(p.st.k) : reinterpret_cast<uint32_t *>(p.mir.k8);
            uint32_t *v8 = toStore8 ? static_cast<uint32_t *>(p.st.v) : reinterpret_cast<uint32_t *>(p.mir.v8);
            float *ks = toStore8 ? p.st.ks : p.mir.ks, *vs = toStore8 ? p.st.vs : p.mir.vs;
            if (!toStore8 && dst >= p.mir.maxRows * p.nKV) {
                if (lane == 0) atomicOr(p.err, kDevErrRowBound);
            } else {
                if (lane == 0) {
                    ks[dst] = sk;
                    vs[dst] = sv;
                }
                auto q8 = [](float x, float sc) -> int {
                    const int qv = __float2int_rn(__fdiv_rn(x, sc));
                    return qv < -128 ? -128 : (qv > 127 ? 127 : qv);
                };
#pragma unroll
                for (int u = 0; u < MAXV; ++u) {
                    if (!active[u]) continue;
                    const uint32_t i4 = lane + 32u * u;
                    auto pack = [&](float4 &x, float sc) -> uint32_t {
                        const int a = q8(x.x, sc), b = q8(x.y, sc), c = q8(x.z, sc), d = q8(x.w, sc);
                        if (toStore8)  // attention over an int8 store sees what the store holds
                            x = make_float4(static_cast<float>(a) * sc, static_cast<float>(b) * sc, static_cast<float>(c) * sc,
                                            static_cast<float>(d) * sc);
                        return (static_cast<uint32_t>(a) & 0xffu) | ((static_cast<uint32_t>(b) & 0xffu) << 8) |
                               ((static_cast<uint32_t>(c) & 0xffu) << 16) | ((static_cast<uint32_t>(d) & 0xffu) << 24);
                    };
                    k8[dst * nvec + i4] = pack(kx[u], sk);
                    v8[dst * nvec + i4] = pack(vx[u], sv);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < MAXV; ++u) {
            if (!active[u]) continue;
            const size_t at = rh * nvec + lane + 32u * u;
            if (fresh && p.st.kind == 0) {
                static_cast<float4 *>(p.st.k)[at] = kx[u];
                static_cast<float4 *>(p.st.v)[at] = vx[u];
            } else if (fresh && p.st.kind == 1) {
                static_cast<uint2 *>(p.st.k)[at] = half4(kx[u]);
                static_cast<uint2 *>(p.st.v)[at] = half4(vx[u]);
            }
            if (p.k16 != nullptr) {
                p.k16[at] = half4(kx[u]);
                p.v16[at] = half4(vx[u]);
            }
        }
    }
}

struct PrefillF16Params {
    float *out;        // [seqLen][nHeads][128] f32
    uint32_t seqLen, nHeads, nKV, group;
    uint32_t cachePos;  // query row r sits at position cachePos + r and sees K/V rows [0, cachePos + r]
    uint32_t nQTiles;   // query blocks of itemRows rows
    uint32_t itemRows;  // 256: two query tiles per work item; 128: one
    uint32_t split;     // one-tile items whose KV tiles the two halves of the block share (even / odd)
    float scaleLog2;   // invSqrt * log2(e)
    unsigned int *err;
    unsigned int *workCounter;  // zero at launch; item gridDim.x + n goes to the n-th request
    uint32_t totalItems;        // nQTiles * nHeads (query block, head) pairs, heavy blocks first
    uint32_t out32;             // out is 32-byte aligned: rows can be written with 32-byte stores
#ifdef TC_TRACE
    unsigned long long *trace;  // [8 roles][64 steps][4 stamps] of block 0
#endif
};

#ifdef TC_TRACE
unsigned long long *g_pfTrace = nullptr;
__device__ __forceinline__ unsigned long long pfTime() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
#define PF_BLK(k) do { if (p.trace) p.trace[8u * 64u * 4u + item * 8u + (k)] = pfTime(); } while (0)
#define PF_STAMP(role, step, k) do { if (p.trace && item == 0u && (step) < 64u) p.trace[((role) * 64u + (step)) * 4u + (k)] = pfTime(); } while (0)
#else
#define PF_STAMP(role, step, k) do { } while (0)
#define PF_BLK(k) do { } while (0)
#endif

// HD = head_dim (64, 128 or 256): a tile is HD / 64 halves of 64 columns (128 bytes, one swizzle span)
// each.  K and V tiles (64 tokens) have rings of their own: the score products run two tiles ahead of the P.V
// products.  At head_dim 256 one query tile and its 256-column accumulator take the room two tiles take at head_dim 128,
// and the rings are two tiles deep.
template <int HD>
struct PrefillF16Smem {
    static constexpr int kHalves = HD / 64;
    static constexpr int kQTiles = HD > 128 ? 1 : 2;   // query tiles a block holds
    static constexpr int NK = HD > 128 ? 2 : 6, NV = HD > 128 ? 2 : 4;
    static constexpr int kQHalf = kPfBM * 128;         // 16 KB: 128 rows x 64 fp16
    static constexpr int kKvHalf = kPfBN * 128;        // kPfBN rows x 64 fp16
    static constexpr int kQTile = kHalves * kQHalf;    // head_dim 128: 32 KB
    static constexpr int kKvTile = kHalves * kKvHalf;  // head_dim 128: 16 KB
    static constexpr int kQ = 0;
    static constexpr int kK = kQTiles * kQTile;
    static constexpr int kV = kK + NK * kKvTile;
    static constexpr int kBars = kV + NV * kKvTile;
    // qFull, kFull + kEmpty, vFull + vEmpty, sFull[2][2], pFull[2][2], pvDone[2], pvBuf[2][2], qFree[2], itemFull[4],
    // exFull, exRead, sFree[2]
    static constexpr int kNumBars = 1 + 2 * NK + 2 * NV + 4 + 4 + 2 + 4 + 2 + 4 + 2 + 2;
    static constexpr int kTmemSlot = kBars + kNumBars * 8;
    static constexpr int kItemSlots = kTmemSlot + 16;  // four work item indices
    static constexpr int kTotal = kItemSlots + 16 + 1024;
    static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

// Bounded wait: 2^18 polls, each parked for up to 20 us by the hardware.
__device__ __forceinline__ bool pfPoll(uint64_t *bar, uint32_t parity, unsigned int *err, uint32_t bit) {
#pragma unroll 1
    for (uint32_t i = 0; i < (1u << 18); ++i) {
        if (mbarTryWait(bar, parity)) return true;
        // somebody has already given up: what this thread waits for will not come either
        if ((i & 63u) == 63u &&
            (*reinterpret_cast<volatile unsigned int *>(err) & (kDevErrFullWait | kDevErrEmptyWait | kDevErrMmaWait)) != 0u)
            return false;
    }
    atomicOr(err, bit);
    return false;
}
static __device__ __noinline__ bool pfPollCall(uint64_t *bar, uint32_t parity, unsigned int *err, uint32_t bit) {
    return pfPoll(bar, parity, err, bit);
}
// Most waits find their phase complete, a step's chain goes through five of them, and their code sits in the middle of long
// unrolled loops: the first poll stands alone and the loop behind it is a call.  Launch of 4096 rows of 28 / 4 / 128 (rows
// launch included) 139.6 us with a loop that reads the clock, 135.3 with the first poll in front of a short loop,
// 130.0 with that loop as a call; 512 rows behind 3584 49.7, 43.7 and 43.4.
template <bool CALL>
__device__ __forceinline__ bool pfWait(uint64_t *bar, uint32_t parity, unsigned int *err, uint32_t bit) {
    return mbarTryWait(bar, parity) || (CALL ? pfPollCall(bar, parity, err, bit) : pfPoll(bar, parity, err, bit));
}

// one 32-byte store (the address has to be 32-byte aligned)
__device__ __forceinline__ void stGlobalV8(float *dst, float a, float b, float c, float d, float e, float f, float g,
                                           float h) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d),
                 "f"(e), "f"(f), "f"(g), "f"(h)
                 : "memory");
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// A matrix descriptor whose start address is moved by `bytes` (the address field holds
// bytes >> 4 in its low 14 bits; shared memory is far smaller than their range, so the sum
// never carries out of the field).
__device__ __forceinline__ uint64_t descAdvance(uint64_t d, uint32_t bytes) { return d + (bytes >> 4); }

// What one work item covers.  Two-tile items (256 query rows of one head): query tile X (0 = A, 1 = B) holds rows
// m0 + 128 X .. at positions cachePos + row and sees KV tiles 0 .. nX - 1 (the last two or three straddle its diagonal); B
// may lie wholly past the sequence.  Split items (128 query rows): both halves of the block work on the same query
// tile, A on the even KV tiles, B on the odd ones, and put their results together at the end -- a call too short to give
// every SM a two-tile item is bound by the chain of one tile's steps, not by the tensor pipe.
// SHARED: block r of a cluster of C takes KV tiles r, r + C, ... of the item (none, if there are fewer than r + 1); nA, nB and
// nTiles count those.
struct PfItem {
    uint32_t head, kvHead, m0, nA, nB, nTiles;
};
template <bool SHARED>
__device__ __forceinline__ PfItem pfItem(const PrefillF16Params &p, uint32_t item) {
    PfItem it;
    const uint32_t qb = p.nQTiles - 1u - item / p.nHeads;  // heavy query blocks (long causal prefixes) first
    it.head = item % p.nHeads;
    it.kvHead = it.head / p.group;
    it.m0 = qb * p.itemRows;
    auto tilesOf = [&](uint32_t row0) {  // KV tiles the rows row0 .. row0 + 127 of the sequence see
        return (p.cachePos + min(row0 + kPfBM, p.seqLen) + kPfBN - 1u) / kPfBN;
    };
    it.nA = tilesOf(it.m0);
    it.nB = p.itemRows > kPfBM && it.m0 + kPfBM < p.seqLen ? tilesOf(it.m0 + kPfBM) : 0u;
    it.nTiles = max(it.nA, it.nB);
    if constexpr (SHARED) {
        const uint32_t r = clusterRank(), c = clusterSize();
        it.nA = it.nTiles = it.nTiles > r ? (it.nTiles - r + c - 1u) / c : 0u, it.nB = 0u;
    }
    if (p.split) it.nB = it.nTiles / 2u, it.nA = it.nTiles - it.nB;
    return it;
}

// 416 threads: warps 0-3 softmax of query tile A, warps 4-7 softmax of query tile B
// (rows 128 further down), warp 8 TMA producer and scheduler, warps 9 and 10 issue the score
// products of A and B, warps 11 and 12 their P.V products.
//
// One block per SM works through (query block, head) items: its first is blockIdx.x, the following
// ones come from a counter, so the heavy items start first and the light ones fill in behind them.
// The roles walk the item list independently and meet only at the mbarriers, which are never
// initialised again: every ring (K/V stages, score buffers, P.V commits) is indexed by a count that
// runs on from item to item.  So the next item's query tiles load as soon as this item's last score
// product has been issued, its first scores are in TMEM while the softmax threads still write this
// item's output, and tile A moves on while tile B finishes its two extra diagonal tiles.
constexpr int kPfThreads = 416;
//
// SHARED: a cluster works on ONE item and leaves.  What bounds an item alone is the chain of its KV tiles' steps (0.9 us
// each), while SMs stand idle.  Per call, one block -> the cluster that prefillShare picks, rows @ rows in front: 8 / 2 / 128 512 @ 512 /
// 1536 / 3584 17.5 / 25.3 / 41.3 -> 16.4 / 17.7 / 22.6 us, 16 / 2 / 256 25.6 / 39.6 / 67.8 -> 20.9 / 28.3 / 43.4, 14 / 2 / 64 512 @ 3584
// 36.7 -> 24.8, 28 / 4 / 128 100 @ 3000 34.3 -> 20.8.  Putting the results together is what limits it: 3 - 8 us.
template <int HD, bool SHARED>
__global__ void __launch_bounds__(kPfThreads, 1)
prefillF16Kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const PrefillF16Params p) {
    using L = PrefillF16Smem<HD>;
    constexpr int BN = kPfBN;
    constexpr int NC = BN / 32;  // 32-column chunks of a score row
    constexpr uint32_t NK = L::NK, NV = L::NV;
    constexpr bool kCall = HD < 256;     // (a call costs the softmax threads of head_dim 256 spills: 68 -> 79 us)
    constexpr bool kOne = L::kQTiles == 1;  // the second half of the block has nothing to do
    // One query tile is a chain of steps; nothing else fills the tensor pipe while it waits.  Its scores take one buffer, free
    // once they are in the softmax threads' registers, and its probabilities two, so that S(t+1) is computed under the
    // exponentials of tile t and waits for no P.V product: 512 rows behind 3000 of 16 / 2 / 256 67.7 -> 58.6 us, 2000 rows of
    // 16 / 4 / 256 55.3 -> 51.0.  With two query tiles the chains fill each other's gaps, and the two waits more per
    // step cost more than that (4096 rows of 28 / 4 / 128 130 -> 137).
    constexpr bool kAhead = kOne;
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kBars);
    uint64_t *qFull = bars, *kFull = bars + 1, *kEmpty = kFull + NK, *vFull = kEmpty + NK, *vEmpty = vFull + NV,
             *sFull = vEmpty + NV /* [x][b] */, *pFull = sFull + 4 /* [x][b] */, *pvDone = pFull + 4 /* [x] */,
             *pvBuf = pvDone + 2 /* [x][b] */, *qFree = pvBuf + 4 /* [x] */, *itemFull = qFree + 2 /* [4] */,
             *exFull = itemFull + 4, *exRead = exFull + 1, *sFree = exRead + 1 /* [x] */;
    uint32_t *tmemSlot = reinterpret_cast<uint32_t *>(smem + L::kTmemSlot);
    volatile uint32_t *itemSlots = reinterpret_cast<volatile uint32_t *>(smem + L::kItemSlots);  // [4]
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;
    const bool split = !kOne && p.split != 0;
    const uint32_t rank = SHARED ? clusterRank() : 0u, share = SHARED ? clusterSize() : 1u;  // KV tile j of the block: share j + rank
    // what a softmax thread hands to the cluster: its row's maximum and sum over the block's tiles, the weights of the halves'
    // accumulators
    float rowM = kNegBig, rowL = 0.0f, rowW = 1.0f, rowW2 = 0.0f;
    bool rowBoth = false, rowAny = false;

    if (threadIdx.x == 0) {
        mbarInit(qFull, 1);
        // a K (V) tile is released by the score (P.V) warps of the query tiles that it serves
        const uint32_t users = kOne || split ? 1u : 2u;
        for (uint32_t s = 0; s < NK; ++s) {
            mbarInit(&kFull[s], 1);
            mbarInit(&kEmpty[s], users);
        }
        for (uint32_t s = 0; s < NV; ++s) {
            mbarInit(&vFull[s], 1);
            mbarInit(&vEmpty[s], users);
        }
        for (int i = 0; i < 4; ++i) {
            mbarInit(&sFull[i], 1);
            mbarInit(&pFull[i], 4);  // one arrival per warp
            mbarInit(&pvBuf[i], 1);
            mbarInit(&itemFull[i], 1);
        }
        for (int x = 0; x < 2; ++x) {
            mbarInit(&sFree[x], 4);  // one arrival per warp
            mbarInit(&pvDone[x], 1);
        }
        mbarInit(&qFree[0], 1);  // score warp X is done with the query tiles
        mbarInit(&qFree[1], 1);
        mbarInit(exFull, 2 * kPfBM);  // split items: every softmax thread has left its (m, l) / has read the accumulators
        mbarInit(exRead, 2 * kPfBM);
        fenceBarrierInit();
        tmaPrefetchDesc(&tmQ);
        tmaPrefetchDesc(&tmK);
        tmaPrefetchDesc(&tmV);
    }
    if (warp == 0) {
        tmemAlloc(tmemSlot, 512);
        tmemRelinquish();
        tcFenceBefore();
    }
    __syncthreads();
    tcFenceAfter();
    const uint32_t tmemBase = *reinterpret_cast<volatile uint32_t *>(tmemSlot);
    // O of tile X at columns 128 X; S buffer b of tile X at 256 + 128 X + 64 b, its fp16 probabilities over the first 32 of
    // those columns.  kAhead: S at 256, the probabilities behind it in two buffers of 32 columns.

    // The n-th item of this block: the producer publishes it in slot n % 4 (the end of the list as
    // an index past the last item); the other roles pick it up there.
    auto takeItem = [&](uint32_t n, uint32_t &item) -> bool {
        if (!pfWait<kCall>(&itemFull[n & 3u], (n >> 2) & 1u, p.err, kDevErrFullWait)) return false;
        item = itemSlots[n & 3u];
        return item < p.totalItems;
    };

    if (warp == 8) {
        // ------------------------ TMA producer and scheduler ------------------------
        if (lane == 0) {
            uint32_t item = SHARED ? blockIdx.x / share : blockIdx.x, gk = 0, gv = 0;  // gk / gv: K / V tiles requested so far, over all items
            gridDepWait();  // the twins and the work counter come from the launch in front
            gridDepLaunch();
            itemSlots[0] = item;
            mbarArrive(&itemFull[0]);
            bool ok = true;
            auto requestK = [&](uint32_t kvHead, uint32_t j) {
                const uint32_t s = gk % NK;
                if (gk >= NK && !pfWait<kCall>(&kEmpty[s], ((gk / NK) - 1u) & 1u, p.err, kDevErrEmptyWait)) return false;
                mbarExpectTx(&kFull[s], L::kKvTile);
#pragma unroll
                for (int h = 0; h < L::kHalves; ++h)
                    tmaLoad3D(smem + L::kK + s * L::kKvTile + h * L::kKvHalf, &tmK, &kFull[s], 64 * h, kvHead, (share * j + rank) * BN);
                ++gk;
                return true;
            };
            auto requestV = [&](uint32_t kvHead, uint32_t j) {
                const uint32_t s = gv % NV;
                if (gv >= NV && !pfWait<kCall>(&vEmpty[s], ((gv / NV) - 1u) & 1u, p.err, kDevErrEmptyWait)) return false;
                mbarExpectTx(&vFull[s], L::kKvTile);
#pragma unroll
                for (int h = 0; h < L::kHalves; ++h)
                    tmaLoad3D(smem + L::kV + s * L::kKvTile + h * L::kKvHalf, &tmV, &vFull[s], 64 * h, kvHead, (share * j + rank) * BN);
                ++gv;
                return true;
            };
            for (uint32_t n = 0; ok && item < p.totalItems; ++n) {
                const PfItem it = pfItem<SHARED>(p, item);
                if (SHARED && it.nTiles == 0u) break;  // (nothing is loaded: the block's part of the cluster's end is all there is)
                PF_BLK(0);
#ifdef TC_TRACE
                if (p.trace) { unsigned sm; asm("mov.u32 %0, %%smid;" : "=r"(sm)); p.trace[8u * 64u * 4u + item * 8u + 6] = sm; }
#endif
                // the query tiles are free once the score warps have issued the last product of the previous item and
                // those products are complete
                if (n > 0)
                    ok = pfWait<kCall>(&qFree[0], (n - 1u) & 1u, p.err, kDevErrEmptyWait) &&
                         (kOne || pfWait<kCall>(&qFree[1], (n - 1u) & 1u, p.err, kDevErrEmptyWait));
                if (!ok) break;
                const int qTiles = kOne || split ? 1 : 2;
                mbarExpectTx(qFull, qTiles * L::kQTile);
                for (int x = 0; x < qTiles; ++x)
#pragma unroll
                    for (int h = 0; h < L::kHalves; ++h)
                        tmaLoad3D(smem + L::kQ + x * L::kQTile + h * L::kQHalf, &tmQ, qFull, 64 * h, it.head,
                                  it.m0 + x * kPfBM);
                ok = requestK(it.kvHead, 0) && (it.nTiles < 2u || requestK(it.kvHead, 1));
                // The next item is drawn late -- with the third last tile request, some six tiles before
                // the consumers finish this item -- so that the blocks which finish first take the
                // heavier of the remaining items.
                const uint32_t drawAt = it.nTiles >= 3u ? it.nTiles - 3u : 0u;
                uint32_t drawn = 0, flags = 0;
                for (uint32_t j = 0; ok && j < it.nTiles; ++j) {
                    if (!SHARED && j == drawAt) {
                        flags = *reinterpret_cast<volatile unsigned int *>(p.err);
                        drawn = gridDim.x + atomicAdd(p.workCounter, 1u);
                    }
                    ok = (j + 2u >= it.nTiles || requestK(it.kvHead, j + 2u)) && requestV(it.kvHead, j);
                }
                if (!ok) break;
                // a wait that ran out anywhere ends the launch: the flag is the caller's to read
                constexpr unsigned int kWaitBits = kDevErrFullWait | kDevErrEmptyWait | kDevErrMmaWait;
                const uint32_t next = SHARED || (flags & kWaitBits) != 0u ? p.totalItems : drawn;
                itemSlots[(n + 1u) & 3u] = next;
                mbarArrive(&itemFull[(n + 1u) & 3u]);
                item = next;
            }
            // the last release of every slot has to have arrived before the block leaves
            for (uint32_t back = 0; ok && back < NK && back < gk; ++back) {
                const uint32_t g = gk - 1u - back;
                ok = pfWait<kCall>(&kEmpty[g % NK], (g / NK) & 1u, p.err, kDevErrEmptyWait);
            }
            for (uint32_t back = 0; ok && back < NV && back < gv; ++back) {
                const uint32_t g = gv - 1u - back;
                ok = pfWait<kCall>(&vEmpty[g % NV], (g / NV) & 1u, p.err, kDevErrEmptyWait);
            }
        }
    } else if (warp >= 9) {
        // ------------------------------- MMA issuers -------------------------------
        // The score products and the P.V products of a query tile have an issuing warp each, so that no wait stands in front
        // of the other tile's products: warp 9 + X issues S_X(t) = Q_X K^T (M128 N64
        // K16 x8), warp 11 + X issues O_X += P_X(t) V (A from TMEM, B = V MN-major from shared
        // memory, K16 x4).  t counts the tiles of X over all items; tile t uses score buffer t % 2,
        // and S_X(t+2) goes into the buffer P_X(t) occupies: the score warp waits for the commit of
        // that P.V product (pvBuf) before it issues.  kAhead: for the softmax threads to have read S(t-1) (sFree).
        // All 32 lanes run this warp-uniform code; the elected one executes the tcgen05 instructions.
        const uint32_t x = (warp - 9u) & 1u;
        const bool pvRole = warp >= 11u;
        constexpr uint32_t idQK = umaInstrDescF16(kPfBM, BN, 0, 0);
        constexpr uint32_t idPV = umaInstrDescF16(kPfBM, HD, 0, 1);
        const uint64_t dQ = umaSmemDesc(smemAddr(smem + L::kQ + (split ? 0u : x) * L::kQTile), 16, 1024);
        const uint64_t dK0 = umaSmemDesc(smemAddr(smem + L::kK), 16, 1024);
        const uint64_t dV0 = umaSmemDesc(smemAddr(smem + L::kV), L::kKvHalf, 1024);
        const uint32_t tO = tmemBase + 128u * x, tS0 = tmemBase + 256u + 128u * x;
        uint32_t g = 0, t = 0, item = 0;  // K (V) tiles of the items done, tiles of X done, over all items
        bool ok = !(kOne && x == 1u);
        for (uint32_t n = 0; ok && takeItem(n, item); ++n) {
            const PfItem it = pfItem<SHARED>(p, item);
            if (SHARED && it.nTiles == 0u) break;
            const uint32_t myTiles = x == 0 ? it.nA : it.nB;
            // A split item's warps look at their own KV tiles only.  In a two-tile item every tile is released by both
            // query tiles' warps, also the ones past a tile's diagonal -- but only after it has been filled: a warp with
            // nothing to do must not run ahead and hand in the release of a later round, or the barrier would complete
            // without the warp that still reads the slot.
            const uint32_t j0 = split ? x : 0u, step = split ? 2u : 1u;
            uint32_t tt = t;
            for (uint32_t j = j0; ok && j < it.nTiles; j += step, ++tt) {
                const uint32_t gg = g + j;
                const bool mine = split || j < myTiles;
                if (!pvRole) {
                    const uint32_t s = gg % NK;
                    if (mine && j == j0) ok = pfWait<kCall>(qFull, n & 1u, p.err, kDevErrFullWait);
                    if (lane == 0) PF_STAMP(2u + x, j, 0);
                    ok = ok && pfWait<kCall>(&kFull[s], (gg / NK) & 1u, p.err, kDevErrFullWait);
                    if (mine) {
                        if (kAhead) {
                            if (ok && tt >= 1u) ok = pfWait<kCall>(&sFree[x], (tt - 1u) & 1u, p.err, kDevErrMmaWait);
                        } else if (ok && tt >= 2u) {
                            ok = pfWait<kCall>(&pvBuf[2u * x + (tt & 1u)], ((tt - 2u) >> 1) & 1u, p.err, kDevErrMmaWait);
                        }
                        if (!ok) break;
                        tcFenceAfter();
                        const uint64_t dK = descAdvance(dK0, s * L::kKvTile);
                        if (electOne()) {
#pragma unroll
                            for (uint32_t ks = 0; ks < HD / 16; ++ks) {
                                // k step ks: dims 16 ks .. +15 = 32 bytes inside the (ks >> 2)-th 64-dim half
                                umaMmaSS(tS0 + (kAhead ? 0u : 64u * (tt & 1u)), descAdvance(dQ, (ks >> 2) * L::kQHalf + (ks & 3u) * 32u),
                                         descAdvance(dK, (ks >> 2) * L::kKvHalf + (ks & 3u) * 32u), idQK, ks > 0 ? 1u : 0u);
                            }
                            umaCommit(&sFull[kAhead ? x : 2u * x + (tt & 1u)]);
                            // the item's last score product: the query tiles may be replaced once it is complete
                            if (tt + 1u == t + myTiles) umaCommit(&qFree[x]);
                            umaCommit(&kEmpty[s]);
                            PF_STAMP(2u + x, j, 2);
                        }
                    } else if (ok && electOne()) {
                        umaCommit(&kEmpty[s]);
                    }
                    __syncwarp();
                } else {
                    const uint32_t s = gg % NV;
                    ok = pfWait<kCall>(&vFull[s], (gg / NV) & 1u, p.err, kDevErrFullWait);
                    if (mine) {
                        if (lane == 0) PF_STAMP(4u + x, j, 0);
                        ok = ok && pfWait<kCall>(&pFull[2u * x + (tt & 1u)], (tt >> 1) & 1u, p.err, kDevErrMmaWait);
                        if (lane == 0) PF_STAMP(4u + x, j, 1);
                        if (!ok) break;
                        tcFenceAfter();
                        const uint64_t dV = descAdvance(dV0, s * L::kKvTile);
                        const uint32_t tP = tS0 + (kAhead ? 64u + 32u * (tt & 1u) : 64u * (tt & 1u));
                        if (electOne()) {
#pragma unroll
                            for (uint32_t ks = 0; ks < BN / 16; ++ks)  // 16 tokens per step: 8 columns of fp16 P, 2 KB of V
                                umaMmaTS(tO, tP + ks * 8u, descAdvance(dV, ks * 2048u), idPV, (tt > t || ks > 0) ? 1u : 0u);
                            umaCommit(&pvBuf[2u * x + (tt & 1u)]);
                            umaCommit(&pvDone[x]);
                            umaCommit(&vEmpty[s]);
                            PF_STAMP(4u + x, j, 2);
                        }
                    } else if (ok && electOne()) {
                        umaCommit(&vEmpty[s]);
                    }
                    __syncwarp();
                }
            }
            // A half without tiles still hands in its phase of qFree, one per item -- but only behind the item's last
            // K tile: the producer fills that tile after it has looked at the previous phase, so this warp cannot
            // complete two phases before the producer has seen the first (a parity wait cannot tell those apart).
            // (A split item without odd tiles has one tile: its own full barrier stands for the last K tile.)
            if (!pvRole && myTiles == 0u && ok) {
                if (split) ok = pfWait<kCall>(&kFull[g % NK], (g / NK) & 1u, p.err, kDevErrFullWait);
                if (ok && electOne()) umaCommit(&qFree[x]);
                __syncwarp();
            }
            t += myTiles;
            g += it.nTiles;
        }
        if (pvRole && ok) {
            // nobody waits for the last two buffer commits; they have to land before the block leaves
            for (uint32_t tt = t >= 2u ? t - 2u : 0u; tt < t; ++tt)
                if (!pfWait<kCall>(&pvBuf[2u * x + (tt & 1u)], (tt >> 1) & 1u, p.err, kDevErrMmaWait)) break;
        }
    } else {
        // --------------------------------- softmax ---------------------------------
        const uint32_t x = warp >> 2;                         // which query tile this warpgroup owns
        const uint32_t row = (warp & 3u) * 32u + lane;        // row of that tile = TMEM lane
        const uint32_t laneBase = ((warp & 3u) * 32u) << 16;  // TMEM lane field
        const uint32_t tileRow0 = split ? 0u : x * kPfBM;     // the tile's first row inside the item
        const uint32_t rowInBlock = tileRow0 + row;
        const uint32_t tO = tmemBase + 128u * x;
        // split items: (m, l) of a half's rows, in the room of the query tile that they do not have
        float2 *exch = reinterpret_cast<float2 *>(smem + L::kQ + (kOne ? 0 : L::kQTile));
        uint32_t t = 0, item = 0;  // tiles of X done over all items
        bool ok = true;
        for (uint32_t n = 0; ok && takeItem(n, item); ++n) {
            const PfItem it = pfItem<SHARED>(p, item);
            const uint32_t m0 = it.m0, head = it.head;
            const uint32_t rq = m0 + rowInBlock;  // query position
            const uint32_t myTiles = x == 0 ? it.nA : it.nB;
            if (SHARED && it.nTiles == 0u) break;
            if (myTiles == 0 && !split) continue;
            float m = kNegBig, l = 0.0f;
            for (uint32_t j = 0; j < myTiles; ++j) {
                const uint32_t tt = t + j, b = tt & 1u;
                const uint32_t kt = share * (split ? 2u * j + x : j) + rank;  // KV tile
                const uint32_t tS = tmemBase + 256u + 128u * x + (kAhead ? 0u : 64u * b), tP = kAhead ? tS + 64u + 32u * b : tS;
                if (row == 0) PF_STAMP(x, j, 0);
                if (!pfWait<kCall>(&sFull[kAhead ? x : 2u * x + b], (kAhead ? tt : tt >> 1) & 1u, p.err, kDevErrMmaWait)) {
                    ok = false;
                    break;
                }
                if (row == 0) PF_STAMP(x, j, 1);
                if (row == 0 && x == 0 && j == 0) PF_BLK(2);
                tcFenceAfter();
                uint32_t r[NC][32];  // the BN scores of this row
#pragma unroll
                for (int c = 0; c < NC; ++c) tmemLd32(tS + laneBase + 32u * c, r[c]);
                tmemLdWait();
                if (kAhead) {
                    tcFenceBefore();
                    __syncwarp();
                    if (lane == 0) mbarArrive(&sFree[x]);  // the next tile's scores may be written
                }
                if (row == 0 && x == 0) PF_STAMP(6u, j, 0);
                if (BN * kt + (BN - 1u) > p.cachePos + m0 + tileRow0) {
                    // causal edge (the tile reaches past the position of this tile's first row): token
                    // 64 kt + c is visible iff it is not past the query position; relative to the item's
                    // first row that is 64 kt - (cachePos + m0) + c <= rowInBlock
                    const int32_t first = static_cast<int32_t>(BN * kt) - static_cast<int32_t>(p.cachePos + m0);
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (first + c * 32 + i > static_cast<int32_t>(rowInBlock)) r[c][i] = 0xff800000u;  // -inf
                }
                float mxs[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int i = 0; i < 32; i += 8)
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            mxs[u] = max3(mxs[u], __uint_as_float(r[c][i + 2 * u]), __uint_as_float(r[c][i + 2 * u + 1]));
                const float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])) * p.scaleLog2;  // scale > 0: max commutes with it
                const float mNew = mx > m + kPfLazyLog2 ? mx : m;
                const bool rescale = j > 0 && __any_sync(0xffffffffu, mNew != m);
                float alpha = 1.0f;  // (without a rescale m stays: l is 0 in the first step)
                if (row == 0 && x == 0) PF_STAMP(6u, j, 1);
                // O may only be touched between two of its PV products: the previous one has to be
                // complete (the next one cannot start before this thread publishes P).  The last
                // step takes the wait in any case: a parity wait can only tell the current phase from
                // the one before it, and the final wait below must not find the barrier two behind.
                // (pvDone completes one phase per tile, so its parity follows the running count.)
                if (j > 0 && (rescale || j + 1u == myTiles)) {
                    if (!pfWait<kCall>(&pvDone[x], (tt - 1u) & 1u, p.err, kDevErrMmaWait)) {
                        ok = false;
                        break;
                    }
                    tcFenceAfter();
                }
                if (rescale) {
                    alpha = fastExp2(m - mNew);
#pragma unroll 1
                    for (uint32_t c = 0; c < HD / 32; ++c) {
                        uint32_t o[32];
                        tmemLd32(tO + laneBase + c * 32u, o);
                        tmemLdWait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmemSt32(tO + laneBase + c * 32u, o);
                    }
                    tmemStWait();
                }
                m = mNew;
                if (kAhead) {
                    // the buffer's last probabilities, those of tile t - 2, have been multiplied (long ago as a rule)
                    if (tt >= 2u && !pfWait<kCall>(&pvBuf[2u * x + b], ((tt - 2u) >> 1) & 1u, p.err, kDevErrMmaWait)) {
                        ok = false;
                        break;
                    }
                    tcFenceAfter();
                }
                // probabilities as fp16 pairs: the A operand of the PV product
                // (every score of the row is already in registers)
                // Pairs of elements with packed f32x2 arithmetic (scale-and-shift, row sum).  Evaluating
                // part of the exponentials on the FMA pipe (round-to-integer trick + cubic) was measured
                // at 25 / 50 / 75 % of the pairs: 716 / 699 / 694 TFLOP/s against 732 with all of them on
                // the special-function unit; a second implementation (magic-constant integer split, cubic
                // with relative error 7.5e-5, exponent patched by an integer add, selected per pair at run
                // time) lost a fifth from 0 to 4 of every 4 pairs.  Exponentials of fp16 PAIRS
                // (ex2.approx.f16x2 on the rounded exponent, row sum over fp16 partial sums) pass the
                // parity tests but are slower too: 673 TFLOP/s.  Per 64-token step a softmax thread is busy
                // for 0.9 us, 0.8 of them in these two loops; more instructions cost time in proportion,
                // whichever pipe they run on.
                const float2 scale2 = make_float2(p.scaleLog2, p.scaleLog2), negM2 = make_float2(-m, -m);
                float psum = 0.0f;
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    uint32_t h[16];
                    {
                        float2 sum2 = make_float2(0.0f, 0.0f);
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 x2 = __ffma2_rn(make_float2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])),
                                                         scale2, negM2);
                            const float2 p2 = make_float2(fastExp2(x2.x), fastExp2(x2.y));
                            sum2 = __fadd2_rn(sum2, p2);
                            h[i] = packHalf2(p2.x, p2.y);
                        }
                        psum += sum2.x + sum2.y;
                    }
                    tmemSt16(tP + laneBase + c * 16u, h);
                    if (row == 0 && x == 0) PF_STAMP(6u, j, 2 + c);
                }
                l = l * alpha + psum;
                tmemStWait();
                tcFenceBefore();
                __syncwarp();
                if (lane == 0) mbarArrive(&pFull[2u * x + b]);
                if (row == 0) PF_STAMP(x, j, 2);
                if (row == 0 && j + 1u == myTiles) PF_BLK(3u + x);
            }
            ok = ok && (myTiles == 0 || pfWait<kCall>(&pvDone[x], (t + myTiles - 1u) & 1u, p.err, kDevErrMmaWait));
            if (!ok) break;
            // Split items: each half leaves (m, l) of its rows for the other one and stores half of the dims, out of both
            // accumulators (they lie in the same TMEM lanes).
            float inv, wOther = 0.0f;
            bool both = false;
            if (split) {
                exch[x * kPfBM + row] = make_float2(m, l);
                tcFenceBefore();
                mbarArrive(exFull);
                ok = pfWait<kCall>(exFull, n & 1u, p.err, kDevErrMmaWait);
                if (!ok) break;
                tcFenceAfter();
                const float2 o = exch[(x ^ 1u) * kPfBM + row];
                const float M = fmaxf(m, o.x), wMine = fastExp2(m - M);
                wOther = fastExp2(o.x - M);
                const float lAll = fmaf(wMine, l, wOther * o.y);
                if constexpr (SHARED) {
                    rowM = M, rowL = lAll, rowW = wMine, rowW2 = wOther;
                    rowBoth = it.nB != 0u, rowAny = true;
                    t += myTiles;
                    continue;
                }
                inv = lAll > 0.0f ? 1.0f / lAll : 0.0f;
                wOther *= inv;
                inv *= wMine;
                both = it.nB != 0u;
            } else {
                tcFenceAfter();
                if constexpr (SHARED) {
                    rowM = m, rowL = l, rowAny = true;
                    t += myTiles;
                    continue;
                }
                inv = l > 0.0f ? 1.0f / l : 0.0f;
            }
            float *orow = p.out + (static_cast<size_t>(rq) * p.nHeads + head) * HD;
            // this half's 32-column chunks
            constexpr uint32_t kChunks = HD / 32;
            const uint32_t c0 = split ? x * (kChunks / 2) : 0u, c1 = split ? c0 + kChunks / 2 : kChunks;
            if (split && x == 1u && !both) inv = 0.0f;  // no odd tiles: accumulator B was never written
#pragma unroll 1
            for (uint32_t c = c0; c < c1; ++c) {
                uint32_t o[32];
                if (split && x == 1u && !both) {
                    // everything is in accumulator A
                    tmemLd32(tmemBase + laneBase + c * 32u, o);
                    tmemLdWait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * wOther);
                } else if (both) {
                    uint32_t o2[32];
                    tmemLd32(tO + laneBase + c * 32u, o);
                    tmemLd32(tmemBase + 128u * (x ^ 1u) + laneBase + c * 32u, o2);
                    tmemLdWait();
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        o[i] = __float_as_uint(fmaf(__uint_as_float(o2[i]), wOther, __uint_as_float(o[i]) * inv));
                } else {
                    tmemLd32(tO + laneBase + c * 32u, o);
                    tmemLdWait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * inv);
                }
                if (rq < p.seqLen && !p.out32) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        *reinterpret_cast<float4 *>(orow + c * 32 + 4 * i) =
                                make_float4(__uint_as_float(o[4 * i]), __uint_as_float(o[4 * i + 1]),
                                            __uint_as_float(o[4 * i + 2]), __uint_as_float(o[4 * i + 3]));
                } else if (rq < p.seqLen) {
                    // 32 bytes per store: a thread owns its row, so a warp's store touches 32 rows, and
                    // whole sectors halve the number of transactions against 16-byte stores
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        stGlobalV8(orow + c * 32 + 8 * i, __uint_as_float(o[8 * i]), __uint_as_float(o[8 * i + 1]),
                                   __uint_as_float(o[8 * i + 2]), __uint_as_float(o[8 * i + 3]),
                                   __uint_as_float(o[8 * i + 4]), __uint_as_float(o[8 * i + 5]),
                                   __uint_as_float(o[8 * i + 6]), __uint_as_float(o[8 * i + 7]));
                }
            }
            if (split) {
                // the next item's first P.V product may overwrite an accumulator once both halves have read it
                tcFenceBefore();
                mbarArrive(exRead);
                ok = pfWait<kCall>(exRead, n & 1u, p.err, kDevErrMmaWait);
            }
            if (threadIdx.x == 0) PF_BLK(5);
            t += myTiles;
        }
    }
    if constexpr (SHARED) {
        // Every block leaves its accumulators (relative to its own maximum), maxima and sums where its tiles were, and block o of the
        // cluster puts the o-th share of the rows together, reading the others' memory row by row.  (Written into the owner's
        // memory instead, a thread its row, 16 bytes at a time: 3 / 6 / 11 us at head_dim 64 / 128 / 256.)  Every thread takes
        // part in the two barriers, whatever became of its waits.
        constexpr uint32_t kRowBytes = HD * 4 + 16;  // (threads of a warp store different rows)
        constexpr uint32_t kAt = kOne ? 0 : L::kK;   // (in split items the halves exchange through the second query tile's room)
        static_assert(kAt + kPfBM * (kRowBytes + 12) <= L::kBars, "the tiles' room");
        const uint32_t stage = smemAddr(smem + kAt), stageMl = stage + kPfBM * kRowBytes;
        float *weights = reinterpret_cast<float *>(smem + kAt + kPfBM * (kRowBytes + 8));  // [block][row of this block's share]
        const uint32_t x = warp >> 2, row = (warp & 3u) * 32u + lane;
        if (warp < (kOne ? 4u : 8u)) {
            const uint32_t laneBase = ((warp & 3u) * 32u) << 16;
            if (x == 0u) asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(stageMl + row * 8u), "f"(rowM), "f"(rowL) : "memory");
            constexpr uint32_t kChunks = HD / 32;
            const uint32_t c0 = split ? x * (kChunks / 2) : 0u, c1 = split ? c0 + kChunks / 2 : kChunks;
            const uint32_t tMine = tmemBase + 128u * x, tOther = tmemBase + 128u * (x ^ 1u);
            // (block-uniform: a block without tiles has nothing in its accumulators; without odd tiles everything is in A)
            const bool onlyOther = split && x == 1u && !rowBoth;
            if (__all_sync(0xffffffffu, rowAny)) {
#pragma unroll 1
                for (uint32_t c = c0; c < c1; ++c) {
                    uint32_t o[32];
                    tmemLd32((onlyOther ? tOther : tMine) + laneBase + c * 32u, o);
                    if (rowBoth) {
                        uint32_t o2[32];
                        tmemLd32(tOther + laneBase + c * 32u, o2);
                        tmemLdWait();
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            o[i] = __float_as_uint(fmaf(__uint_as_float(o2[i]), rowW2, __uint_as_float(o[i]) * rowW));
                    } else {
                        tmemLdWait();
                        const float w = onlyOther ? rowW2 : rowW;
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * w);
                    }
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + row * kRowBytes + (c * 32u + i) * 4u),
                                     "r"(o[i]), "r"(o[i + 1]), "r"(o[i + 2]), "r"(o[i + 3])
                                     : "memory");
                }
            }
        }
        clusterSync();
        const uint32_t rows = kPfBM / share, item = blockIdx.x / share;
        const uint32_t head = item % p.nHeads, first = (p.nQTiles - 1u - item / p.nHeads) * p.itemRows;
        constexpr uint32_t V4 = HD / 4;
        // Every lane's access to another block's memory is a request of its own, one per cycle and SM (with the maxima and sums
        // read beside each value, and this block's own results the same way, this took 8.4 us at head_dim 256): the weights of
        // the blocks come first, once per row.
        if (threadIdx.x < rows) {
            float2 ml[8];
            float M = kNegBig, l = 0.0f;
#pragma unroll
            for (uint32_t b = 0; b < 8u; ++b) {
                ml[b] = make_float2(kNegBig, 0.0f);
                if (b < share)
                    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];"
                                 : "=f"(ml[b].x), "=f"(ml[b].y) : "r"(mapRank(stageMl + (rank * rows + threadIdx.x) * 8u, b)));
            }
#pragma unroll
            for (uint32_t b = 0; b < 8u; ++b) M = fmaxf(M, ml[b].x);
#pragma unroll
            for (uint32_t b = 0; b < 8u; ++b) l = fmaf(fastExp2(ml[b].x - M), ml[b].y, l);
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
            for (uint32_t b = 0; b < 8u; ++b)  // (0: no tile of that block has tokens for the row, or it has no tiles at all)
                if (b < share) weights[b * rows + threadIdx.x] = ml[b].y != 0.0f ? fastExp2(ml[b].x - M) * inv : 0.0f;
        }
        __syncthreads();
        constexpr uint32_t U = 4;  // outputs of a thread on the way together
        const uint32_t total = min(rows, p.seqLen > first + rank * rows ? p.seqLen - first - rank * rows : 0u) * V4;
        for (uint32_t i0 = threadIdx.x; i0 < total; i0 += U * kPfThreads) {
            float4 acc[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t b = 0; b < share; ++b) {
                const uint32_t from = mapRank(stage, b);
                float4 a[U];
#pragma unroll
                for (uint32_t u = 0; u < U; ++u) {
                    const uint32_t i = min(i0 + u * kPfThreads, total - 1u), at = (rank * rows + i / V4) * kRowBytes + i % V4 * 16u;
                    if (b == rank) a[u] = *reinterpret_cast<const float4 *>(smem + kAt + at);
                    else
                        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(a[u].x), "=f"(a[u].y), "=f"(a[u].z), "=f"(a[u].w) : "r"(from + at));
                }
#pragma unroll
                for (uint32_t u = 0; u < U; ++u) {
                    const float w = weights[b * rows + min(i0 + u * kPfThreads, total - 1u) / V4];
                    if (w == 0.0f) continue;
                    acc[u].x = fmaf(w, a[u].x, acc[u].x), acc[u].y = fmaf(w, a[u].y, acc[u].y);
                    acc[u].z = fmaf(w, a[u].z, acc[u].z), acc[u].w = fmaf(w, a[u].w, acc[u].w);
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t i = i0 + u * kPfThreads;
                if (i >= total) break;
                *reinterpret_cast<float4 *>(p.out + (static_cast<size_t>(first + rank * rows + i / V4) * p.nHeads + head) * HD + i % V4 * 4u) = acc[u];
            }
        }
        clusterSync();  // (nobody reads this block's memory any more)
    }
    tcFenceBefore();
    __syncthreads();
    if (warp == 0) {
        tcFenceAfter();
        tmemDealloc(tmemBase, 512);
    }
}

static int f16Map(const void *base, uint32_t hd, uint32_t heads, uint32_t rows, uint32_t boxRows, CUtensorMap *out) {
    TensorMapKey key;
    memset(&key, 0, sizeof(key));
    key.base = base;
    key.rank = 3;
    key.elemBytes = 2;
    key.swizzle = 3;
    key.dims[0] = hd;
    key.dims[1] = heads;
    key.dims[2] = rows;
    key.strides[0] = hd * 2;
    key.strides[1] = static_cast<uint64_t>(heads) * hd * 2;
    key.box[0] = 64;  // 128 bytes: one swizzle span
    key.box[1] = 1;
    key.box[2] = boxRows;
    return getTensorMap(key, out);
}

static size_t prefillScratchBytes(uint32_t seqLen, uint32_t cachePos, uint32_t nHeads, uint32_t nKV, uint32_t hd) {
    // fp16 twins: q [seqLen][nHeads][hd], k and v [cachePos + seqLen][nKV][hd]; each region 1 KB aligned;
    // then the work counter of the attention launch
    auto al = [](size_t x) { return (x + 1023) & ~size_t(1023); };
    return al(static_cast<size_t>(seqLen) * nHeads * hd * 2) +
           2 * al((static_cast<size_t>(cachePos) + seqLen) * nKV * hd * 2) + 1024;  // + the work counter
}

}  // namespace tc

#ifdef TC_TRACE
extern "C" void tc_debug_trace_prefill(unsigned long long *buf) { tc::g_pfTrace = buf; }
#endif

extern "C" {

int tc_attn_prefill_f16_scratch_bytes(uint32_t seqLen, uint32_t cachePos, uint32_t nHeads, uint32_t nKV, uint32_t hd,
                                      size_t *bytes) {
    TC_REQUIRE(bytes != nullptr, TC_EINVAL, "tc_attn_prefill_f16_scratch_bytes: null output");
    TC_REQUIRE(hd == 64 || hd == 128 || hd == 256, TC_EUNSUPPORTED, "tc_attn_prefill_f16: head_dim %u (built for 64, 128 and 256)", hd);
    *bytes = tc::prefillScratchBytes(seqLen, cachePos, nHeads, nKV, hd);
    return TC_OK;
}

}  // extern "C"

namespace tc {

// How many blocks share an item's KV tiles.  All clusters have to be resident at once (2 blocks: 74 clusters, 4: 33, 8: 15).  In 0.1
// us: a step of a block's halves takes 9; putting the blocks' results together takes 20 more than an item's own end, and
// what the rows of a block cost to fetch from the others.
static uint32_t prefillShare(uint32_t items, uint32_t tiles, uint32_t halves, uint32_t hd, const uint32_t *maxClusters) {
    auto cost = [&](uint32_t c) { return (tiles + halves * c - 1u) / (halves * c) * 9u + (c > 1u ? 20u + hd * (c - 1u) / (4u * c) : 0u); };
    uint32_t best = 1;
    for (uint32_t lg = 1; lg <= 3; ++lg)
        if (items <= maxClusters[lg] && cost(1u << lg) < cost(best)) best = 1u << lg;
    return best;
}

template <int HD>
static int launchPrefill(const PrefillF16Params &prm, uint32_t tiles, const CUtensorMap &tmQ, const CUtensorMap &tmK,
                         const CUtensorMap &tmV, cudaStream_t st) {
    constexpr size_t smem = PrefillF16Smem<HD>::kTotal;
    // (the blocks allocate TMEM and set up their barriers while the rows launch drains; the producer waits for it before its
    // first load, nothing else reads its outputs)
    if (prm.itemRows == kPfBM) {
        static ClusterSetup setup;
        const uint32_t *limits = nullptr;
        const int rc = setupCluster(setup, prefillF16Kernel<HD, true>, kPfThreads, smem, &limits);
        if (rc != TC_OK) return rc;
        const uint32_t share = prefillShare(prm.totalItems, tiles, prm.split ? 2u : 1u, HD, limits);
        if (share > 1u)
            return launchDependent(prefillF16Kernel<HD, true>, dim3(prm.totalItems * share), kPfThreads, smem, st, share, tmQ, tmK, tmV, prm);
    }
    static bool attrDone[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attrDone[dev]) {
        TC_CUDA_OK(cudaFuncSetAttribute(prefillF16Kernel<HD, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        attrDone[dev] = true;
    }
    const uint32_t grid = std::min<uint32_t>(prm.totalItems, static_cast<uint32_t>(numSMs()));  // one block per SM
    return launchDependent(prefillF16Kernel<HD, false>, dim3(grid), kPfThreads, smem, st, 1, tmQ, tmK, tmV, prm);
}

int prefillF16(float *q, const PrefillKvStore &src, float *out, void *scratch, size_t scratchBytes, uint32_t seqLen,
               uint32_t cachePos, uint32_t nHeads, uint32_t nKV, uint32_t hd, float invSqrt, const PrefillMirror &mir,
               const PrefillNewRows &nr, cudaStream_t st) {
    const void *kvK = src.k, *kvV = src.v;
    TC_REQUIRE(q && kvK && kvV && out && scratch, TC_EINVAL, "tc_attn_prefill_f16: null pointer");
    TC_REQUIRE(src.kind != 2 || (src.ks && src.vs), TC_EINVAL, "tc_attn_prefill_f16: null scale pointer");
    TC_REQUIRE(hd == 64 || hd == 128 || hd == 256, TC_EUNSUPPORTED, "tc_attn_prefill_f16: head_dim %u (built for 64, 128 and 256)", hd);
    TC_REQUIRE(nKV > 0 && nHeads % nKV == 0, TC_EINVAL, "tc_attn_prefill_f16: nHeads %u not a multiple of nKV %u",
               nHeads, nKV);
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kvK) | reinterpret_cast<uintptr_t>(kvV) |
                 reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(scratch) | reinterpret_cast<uintptr_t>(nr.k) |
                 reinterpret_cast<uintptr_t>(nr.v) | reinterpret_cast<uintptr_t>(nr.cosT) |
                 reinterpret_cast<uintptr_t>(nr.sinT)) & 15u) == 0,
               TC_EINVAL, "tc_attn_prefill_f16: pointers need 16-byte alignment");
    if (seqLen == 0) return TC_OK;
    TC_REQUIRE(static_cast<uint64_t>(cachePos) + seqLen < (1ull << 31), TC_EUNSUPPORTED,
               "tc_attn_prefill_f16: %u + %u rows", cachePos, seqLen);
    // an fp16 store is read in place: only q's twin and the counter live in the scratch
    const size_t need = src.kind == 1 ? prefillScratchBytes(seqLen, 0, nHeads, 0, hd)
                                      : prefillScratchBytes(seqLen, cachePos, nHeads, nKV, hd);
    TC_REQUIRE(scratchBytes >= need, TC_EWORKSPACE, "tc_attn_prefill_f16: scratch of %zu bytes, %zu needed",
               scratchBytes, need);
    TC_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 1023u) == 0, TC_EINVAL,
               "tc_attn_prefill_f16: scratch needs 1024-byte alignment");
    const int sms = numSMs();
    // two query tiles per item keep both softmax warpgroups of a block busy; a call too short to give
    // every SM such an item (a 512-row chunk of a prompt: 2 x nHeads items) is cut into one-tile items
    // (head_dim 256: a block holds one query tile, so its items are always one-tile items)
    const uint32_t itemRows =
            hd == 256 || static_cast<uint64_t>((seqLen + 2 * kPfBM - 1) / (2 * kPfBM)) * nHeads < static_cast<uint64_t>(sms)
                    ? kPfBM
                    : 2 * kPfBM;
    const uint32_t nQTiles = (seqLen + itemRows - 1) / itemRows;
    TC_REQUIRE(static_cast<uint64_t>(nQTiles) * nHeads < (1ull << 31), TC_EUNSUPPORTED,
               "tc_attn_prefill_f16: grid too large");
    auto al = [](size_t x) { return (x + 1023) & ~size_t(1023); };
    const size_t qElems = static_cast<size_t>(seqLen) * nHeads * hd;
    const uint32_t kvRows = cachePos + seqLen;  // the cache rows this call attends over
    const size_t kvElems = static_cast<size_t>(kvRows) * nKV * hd;
    uint8_t *sc = static_cast<uint8_t *>(scratch);
    void *q16 = sc, *k16 = sc + al(qElems * 2), *v16 = sc + al(qElems * 2) + al(kvElems * 2);
    unsigned int *workCounter = reinterpret_cast<unsigned int *>(sc + al(qElems * 2) + 2 * al(kvElems * 2));
    if (src.kind == 1) {
        k16 = const_cast<void *>(kvK);
        v16 = const_cast<void *>(kvV);
        workCounter = reinterpret_cast<unsigned int *>(sc + al(qElems * 2));
    }
    unsigned int *err = devErrorWord();
    TC_REQUIRE(err != nullptr, TC_ECUDA, "tc_attn_prefill_f16: no device error word");
    {
        PrefillRowsParams rp;
        rp.q = q;
        rp.q16 = static_cast<uint2 *>(q16);
        rp.k16 = src.kind == 1 ? nullptr : static_cast<uint2 *>(k16);
        rp.v16 = src.kind == 1 ? nullptr : static_cast<uint2 *>(v16);
        rp.st = src;
        rp.nr = nr;
        rp.mir = mir;
        rp.seqLen = seqLen, rp.cachePos = cachePos, rp.nHeads = nHeads, rp.nKV = nKV;
        rp.err = err, rp.workCounter = workCounter;
        const size_t rowHeads = static_cast<size_t>(src.kind == 1 ? (nr.k != nullptr ? seqLen : 0) : kvRows) * nKV;
        // A short call is a chain of latencies: q has blocks of its own, so that K and V do not wait behind it -- while an SM holds
        // two blocks of each kind (four are resident), and the rows that the store already has are no more than q's.  With the
        // attention launch, every block does both -> apart: 8 / 2 / 128 int8, 60 rows 7.2 -> 6.85 us, 512 behind 512 (256 and 256
        // blocks) 15.5 -> 14.95; 14 / 2 / 64 fp16, 512 behind 512 12.8 -> 12.1.  Beyond the line: 12 / 2 / 128, 512 rows (384 and 128)
        // 12.1 -> 12.5; 28 / 4 / 128, 200 rows (350 and 100) 9.6 -> 9.85; 8 / 2 / 128, 60 behind 500 (30 and 140) 10.7 -> 11.1.  (Two
        // instantiations: with a choice at run time the calls that do both lost 0.1 - 0.2 us.)
        const size_t most = static_cast<size_t>(sms) * 16, qBlocks = (qElems / 8 + 255) / 256, kvBlocks = (rowHeads * 32 + 255) / 256;
        const size_t oldBlocks = ((rowHeads - (nr.k != nullptr ? static_cast<size_t>(seqLen) * nKV : 0)) * 32 + 255) / 256;
        const bool apart = kvBlocks != 0 && std::max(qBlocks, kvBlocks) <= static_cast<size_t>(sms) * 2 && oldBlocks <= qBlocks;
        rp.qBlocks = apart ? static_cast<uint32_t>(qBlocks) : 0u;
        const uint32_t blocks = static_cast<uint32_t>(std::min(apart ? qBlocks + kvBlocks : std::max(qBlocks, kvBlocks), most));
        // (half of L2 at most)
        const size_t oldBytes = (rowHeads - (nr.k != nullptr ? static_cast<size_t>(seqLen) * nKV : 0)) * hd * (src.kind == 2 ? 2 : 8);
        const size_t newBytes = nr.k != nullptr ? static_cast<size_t>(seqLen) * nKV * hd * 8 : 0;
        rp.prefetchBlocks = oldBytes + newBytes + qElems * 4 <= (size_t(64) << 20) ? std::min(blocks, static_cast<uint32_t>(sms)) : 0u;
        static constexpr decltype(&prefillRowsKernel<64, false>) kerns[3][2] = {{prefillRowsKernel<64, false>, prefillRowsKernel<64, true>},
                                                                               {prefillRowsKernel<128, false>, prefillRowsKernel<128, true>},
                                                                               {prefillRowsKernel<256, false>, prefillRowsKernel<256, true>}};
        const int rc = launchDependent(kerns[hd == 64 ? 0 : hd == 128 ? 1 : 2][apart ? 1 : 0], dim3(blocks), 256, 0, st, 1, rp);
        if (rc != TC_OK) return rc;
    }
    CUtensorMap tmQ, tmK, tmV;
    int rc = f16Map(q16, hd, nHeads, seqLen, kPfBM, &tmQ);
    if (rc != TC_OK) return rc;
    rc = f16Map(k16, hd, nKV, kvRows, kPfBN, &tmK);
    if (rc != TC_OK) return rc;
    rc = f16Map(v16, hd, nKV, kvRows, kPfBN, &tmV);
    if (rc != TC_OK) return rc;
    PrefillF16Params prm;
    prm.out = out;
    prm.seqLen = seqLen;
    prm.cachePos = cachePos;
    prm.nHeads = nHeads;
    prm.nKV = nKV;
    prm.group = nHeads / nKV;
    prm.nQTiles = nQTiles;
    prm.itemRows = itemRows;
    prm.split = itemRows == kPfBM && hd != 256 ? 1u : 0u;
    prm.scaleLog2 = invSqrt * kLog2e;
    prm.err = err;
    prm.workCounter = workCounter;
    prm.totalItems = nQTiles * nHeads;
    prm.out32 = (reinterpret_cast<uintptr_t>(out) & 31u) == 0 ? 1u : 0u;
#ifdef TC_TRACE
    prm.trace = tc::g_pfTrace;
#endif
    const uint32_t tiles = (kvRows + kPfBN - 1u) / kPfBN;  // of the heaviest item
    if (hd == 64) return launchPrefill<64>(prm, tiles, tmQ, tmK, tmV, st);
    if (hd == 128) return launchPrefill<128>(prm, tiles, tmQ, tmK, tmV, st);
    return launchPrefill<256>(prm, tiles, tmQ, tmK, tmV, st);
}

static int prefillStore(const float *q, const PrefillKvStore &src, float *out, void *scratch, size_t scratchBytes,
                        uint32_t seqLen, uint32_t cachePos, uint32_t nHeads, uint32_t nKV, uint32_t hd, float invSqrt,
                        const PrefillMirror &mir, tc_stream stream) {
    PrefillNewRows none;
    memset(&none, 0, sizeof(none));
    return prefillF16(const_cast<float *>(q), src, out, scratch, scratchBytes, seqLen, cachePos, nHeads, nKV, hd, invSqrt, mir,
                      none, static_cast<cudaStream_t>(stream));
}

}  // namespace tc

extern "C" {

int tc_attn_prefill_f16(const float *q, const float *kvK, const float *kvV, float *out, void *scratch,
                        size_t scratchBytes, uint32_t seqLen, uint32_t cachePos, uint32_t nHeads, uint32_t nKV,
                        uint32_t hd, float invSqrt, tc_stream stream) {
    tc::PrefillMirror none;
    memset(&none, 0, sizeof(none));
    const tc::PrefillKvStore src = {0, const_cast<float *>(kvK), const_cast<float *>(kvV), nullptr, nullptr};
    return tc::prefillStore(q, src, out, scratch, scratchBytes, seqLen, cachePos, nHeads, nKV, hd, invSqrt, none, stream);
}

int tc_attn_prefill_f16_kvhalf(const float *q, const void *kvK16, const void *kvV16, float *out, void *scratch,
                               size_t scratchBytes, uint32_t seqLen, uint32_t cachePos, uint32_t nHeads, uint32_t nKV,
                               uint32_t hd, float invSqrt, tc_stream stream) {
    tc::PrefillMirror none;
    memset(&none, 0, sizeof(none));
    const tc::PrefillKvStore src = {1, const_cast<void *>(kvK16), const_cast<void *>(kvV16), nullptr, nullptr};
    return tc::prefillStore(q, src, out, scratch, scratchBytes, seqLen, cachePos, nHeads, nKV, hd, invSqrt, none, stream);
}

int tc_attn_prefill_f16_i8(const float *q, const int8_t *k8, const int8_t *v8, const float *ks, const float *vs,
                           float *out, void *scratch, size_t scratchBytes, uint32_t seqLen, uint32_t cachePos,
                           uint32_t nHeads, uint32_t nKV, uint32_t hd, float invSqrt, tc_stream stream) {
    tc::PrefillMirror none;
    memset(&none, 0, sizeof(none));
    const tc::PrefillKvStore src = {2, const_cast<int8_t *>(k8), const_cast<int8_t *>(v8), const_cast<float *>(ks),
                                    const_cast<float *>(vs)};
    return tc::prefillStore(q, src, out, scratch, scratchBytes, seqLen, cachePos, nHeads, nKV, hd, invSqrt, none, stream);
}

int tc_attn_prefill_f16_kv8(const float *q, const float *kvK, const float *kvV, float *out, void *scratch,
                            size_t scratchBytes, uint32_t seqLen, uint32_t cachePos, uint32_t nHeads, uint32_t nKV,
                            uint32_t hd, float invSqrt, int8_t *k8, int8_t *v8, float *ks, float *vs,
                            uint64_t kv8Row, uint64_t kv8MaxRows, tc_stream stream) {
    TC_REQUIRE(k8 && v8 && ks && vs, TC_EINVAL, "tc_attn_prefill_f16_kv8: null pool pointer");
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(k8) | reinterpret_cast<uintptr_t>(v8)) & 3u) == 0, TC_EINVAL,
               "tc_attn_prefill_f16_kv8: k8/v8 need 4-byte alignment");
    if (kv8Row + seqLen > kv8MaxRows) {
        tc::setError("tc_attn_prefill_f16_kv8: rows [%llu, %llu) pass the pool's %llu rows", (unsigned long long) kv8Row,
                     (unsigned long long) kv8Row + seqLen, (unsigned long long) kv8MaxRows);
        return TC_ECONTEXT_FULL;
    }
    tc::PrefillMirror mir;
    mir.k8 = k8, mir.v8 = v8, mir.ks = ks, mir.vs = vs, mir.dstRow = kv8Row, mir.maxRows = kv8MaxRows;
    const tc::PrefillKvStore src = {0, const_cast<float *>(kvK), const_cast<float *>(kvV), nullptr, nullptr};
    return tc::prefillStore(q, src, out, scratch, scratchBytes, seqLen, cachePos, nHeads, nKV, hd, invSqrt, mir, stream);
}

}  // extern "C"
