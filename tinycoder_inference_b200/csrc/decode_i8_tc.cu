// decode_i8_tc.cu -- split-KV decode attention over the int8 store on the 5th-generation
// tensor cores (tcgen05.mma kind::i8, accumulators in TMEM), head_dim 128.
//
// What it replaces: kQ35WarpAttention8Split (+ kAttnCombinePartial) and the eager
// kQ35WarpAttention8 of the reference (include/gpu/GpuQwen35Kernels.hpp:519-581, 641-692):
// score = dot(q, float(k8) * sk) * invSqrt, online softmax with exp2, out = sum p * float(v8) * sv.
//
// Why integer tensor cores in an HBM-bound kernel: at 5..8 q heads per kv head the dequantise +
// FMA work is beyond the CUDA cores at HBM speed, and the mma.sync form of this kernel
// (decode_i8.cu) is bound by the ~770 warp instructions it spends per 32 tokens on unpacking
// bytes into fp16 fragments.  Here the K and V tiles go from TMA straight into the tensor core:
//   * S^T[128 tokens x 32] = K[128 x 128 int8] . Qd^T, where Qd holds each q head as three
//     signed base-128 digit planes (q = 2^e * sum_i d_i 128^-i, 21 bits): the A operand is the K
//     tile exactly as TMA wrote it (K-major, 128-byte swizzle), int32 results in TMEM.
//   * a softmax thread owns one token: it reads its 24 integers (tcgen05.ld), rebuilds the 8
//     scores in f32, applies the row's K scale, exponentiates against a reference point that
//     all threads of the warpgroup share (moved only when a score runs ahead by 2^8), and
//     writes p * sv as a 32-bit fixed-point number per head -- whose four bytes ARE four
//     unsigned base-256 digit planes -- into the B operand tile in shared memory.
//   * O^T[128 dims x 32] = V^T[128 x 128 tokens] . Pd (A = the V tile as stored, MN-major;
//     B unsigned digits): int32 per tile in TMEM, folded into f32 registers (thread = dim)
//     with the tile's scale and reference point.  Integer accumulation never spans more than
//     one 128-token tile.
// Every product is exact; the only roundings are the 21-bit q digits, the 2^-24 fixed-point
// step of p * sv, and the f32 folds -- below the f32 arithmetic noise of the reference.
//
// CTA = one kv head x one token range (grid: chunks, kv heads, sequences), 17 warps:
// warps 0-3 / 4-7 two softmax warpgroups taking alternate tiles (scores -> probabilities only),
// warps 8-11 the fold warpgroup (thread = head dimension: every tile's integer P.V out of TMEM into
// f32 accumulators, so a softmax warpgroup's next tile does not wait for the previous
// one's fold), warp 12 TMA producer (six-stage ring of K, V and their scales), warps 13-16 issue the
// MMAs (score / P.V products of even / odd tiles; one elected thread of each).  Partials leave in the reference's layout for the merge kernel (merge.cu).
//
// What bounds it up to some ten megabytes of rows is a chain of latencies: a softmax warp issues an instruction of its tile every
// five cycles or so, alone on its scheduler or not.  So the loops carry as few as they can: digit planes combine two at a time in
// integers before the conversions, only the q heads there are (NH) are worked on, the fold keeps accumulators per softmax
// warpgroup and rescales them when the reference point moved, one arrival per warp, one barrier wait per tile of a softmax
// thread.  A steady tile takes it 970 cycles (1280 before); the first one, whose reference point has to be agreed on, 0.5 us
// (0.8 with shuffles in place of redux.max).  28 / 4 heads, per layer: 32768 rows 10.95 -> 10.15 us, 4098 rows with an f32 mirror
// 7.2 -> 6.65, 8 sequences of 8192 15.0 -> 14.3, 64 of 512 - 32768 rows 197 -> 190.
#include <cstdlib>

#include "tc_tcgen05.cuh"
#include "decode_cluster.cuh"

namespace tc {

struct DecodeTcParams {
    const float *q;
    float *out;
    const float *ks, *vs;
    const float *appendK, *appendV;  // nullable: [batch][nKV][128] rows to quantise into row len - 1 first
    int8_t *k8w, *v8w;               // the pools, for that row
    float *mirK, *mirV;              // nullable: an f32 store that gets the row verbatim
    const int8_t *nextK8, *nextV8;  // nullable: pools of the next call (L2 prefetch)
    float *pAcc, *pM, *pL;
    uint32_t *tickets;           // nullable: [batch][nKV] arrival counters of the in-kernel merge (zero between calls)
    const uint32_t *devLens;     // nullable
    const uint64_t *devRowBase;  // nullable
    uint64_t rowsPerSeq, totalRows;
    uint32_t lenHost, lenAdd;
    uint32_t nHeads, nKV, group, colBase;
    uint32_t chunkTokens, numChunks;
    uint32_t prefetchRows;
    float invSqrt;
    int directOut;
    int dependent;          // TC_DECODE_PDL: the next grid may start ahead of this one's wait
    int prefetchNext;       // 1: yes, 2: only blocks of more than kLateTiles tiles
    uint32_t earlyStages;   // tiles the producer may request before the dependency wait
    int l2Hints;            // bit 0: own tiles evict_first, bit 1: next pools evict_last
    unsigned int *err;
#ifdef TC_TRACE
    unsigned long long *trace;  // [160 blocks][32 stamps]
#endif
};

#ifdef TC_TRACE
__device__ __forceinline__ unsigned long long gtime() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
#define TC_STAMP(slot) do { if (p.trace) p.trace[(blockIdx.x + gridDim.x * blockIdx.y) * 32 + (slot)] = gtime(); } while (0)
#else
#define TC_STAMP(slot) do { } while (0)
#endif

constexpr int kTcTile = 128;      // tokens per tile = MMA M of the score product
constexpr float kTcLazyLog2 = 8.0f;
constexpr uint32_t kLateTiles = 12;  // blocks of more tiles pull the next call's rows when their own are in

// NWG softmax warpgroups take the tiles round-robin (tile j belongs to warpgroup j % NWG and uses its
// buffer (j / NWG) & 1); NS ring stages.  Warps: [0, 4 NWG) softmax, 4 NWG the TMA producer, then
// four MMA issuers.
template <int NWG, int NS>
struct DecodeTcSmem {
    static constexpr int kThreads = (4 * NWG + 4 + 5) * 32;   // softmax warpgroups, the fold warpgroup, producer, 4 MMA issuers
    static constexpr int kTileBytes = kTcTile * 128;              // K (or V) tile: 128 rows x 128 B
    static constexpr int kStageBytes = 2 * kTileBytes + 1024;     // + 128 K scales + 128 V scales
    static constexpr int kQd = NS * kStageBytes;                  // 32 rows x 128 B digit planes of q
    static constexpr int kP = kQd + 4096;                         // 2 NWG probability tiles of 128 x 32 B
    static constexpr int kRed = kP + 2 * NWG * 4096;              // [NWG warpgroups][4 warps][12] floats
    static constexpr int kHs = kRed + NWG * 4 * 12 * 4;           // head scales [8]
    // per (warpgroup, tile of the warpgroup % 4): reference points [8], tile scale, whether they moved.  Four, not two, slots:
    // scores of tile j wait for the P.V product of tile j - 2 NWG, which waits for the fold of tile j - 4 NWG.
    static constexpr int kMeta = kHs + 64;
    static constexpr int kBars = kMeta + 4 * NWG * 12 * 4;
    // full[NS], empty[NS], sFull[2 NWG], pFull[2 NWG], oFull[2 NWG], oFree[2 NWG], qFull, rowFull
    static constexpr int kNumBars = 2 * NS + 8 * NWG + 2;
    static constexpr int kTmemCols = 128 * NWG;                   // S and O buffers of 32 columns each
    static constexpr int kTmemSlot = kBars + kNumBars * 8;
    static constexpr int kTotal = kTmemSlot + 16 + 1024;
    static_assert(kStageBytes % 1024 == 0, "stages keep the 1024-byte alignment of the 128-byte swizzle");
    static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

// ---- helpers local to this kernel ---------------------------------------------------------
__device__ __forceinline__ uint64_t tcDesc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t swz) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr >> 4) & 0x3fffu);
    d |= static_cast<uint64_t>((lbo >> 4) & 0x3fffu) << 16;
    d |= static_cast<uint64_t>((sbo >> 4) & 0x3fffu) << 32;
    d |= 1ull << 46;
    d |= static_cast<uint64_t>(swz) << 61;  // 2 = 128-byte swizzle, 6 = 32-byte swizzle
    return d;
}
// kind::i8 instruction descriptor: int32 accumulator (c_format 2 at bit 4), a/b format at bits
// 7 / 10 (1 = signed, 0 = unsigned 8-bit), a/b major at bits 15 / 16 (1 = MN-major), N >> 3 at 17,
// M >> 4 at 24.
__host__ __device__ constexpr uint32_t tcIdescI8(uint32_t M, uint32_t N, uint32_t aMN, uint32_t bMN, uint32_t aSigned,
                                                 uint32_t bSigned) {
    return (2u << 4) | (aSigned << 7) | (bSigned << 10) | (aMN << 15) | (bMN << 16) | ((N >> 3) << 17) | ((M >> 4) << 24);
}
__device__ __forceinline__ void tcMmaI8(uint32_t dTmem, uint64_t aDesc, uint64_t bDesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(dTmem),
            "l"(aDesc), "l"(bDesc), "r"(idesc), "r"(accumulate)
            : "memory");
}
__device__ __forceinline__ void tmemLd16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr)
            : "memory");
}
__device__ __forceinline__ void tmemLd8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
// all `threads` threads of named barrier `id` arrive; returns the OR of their predicates
__device__ __forceinline__ bool barOr(uint32_t id, uint32_t threads, bool pred) {
    uint32_t r;
    asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 q, %3, 0;\n\t"
            "bar.red.or.pred p, %1, %2, q;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(r)
            : "r"(id), "r"(threads), "r"(static_cast<uint32_t>(pred))
            : "memory");
    return r != 0;
}
// maximum over the warp (NaN is ignored, as in fmaxf); volatile, or it may end up where only lane 0 uses the result
__device__ __forceinline__ float warpMax(float x) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float i2f(uint32_t x) { return __int2float_rn(static_cast<int>(x)); }

// APPEND: the instantiation for calls that hand in the new token's rows.  It is a kernel of its own
// because the mere presence of that (cold) code -- inlined or called, inside or behind the producer's
// loop -- cost the 7B-shaped batch-1 step 0.5 us; calls without new rows run the other instantiation.
// FOLD: how a sequence's blocks come together: a merge launch (or one block per sequence, which writes the output), the
// last block to arrive (tickets), or a cluster that holds them all and folds through distributed shared memory.
enum class TcFold { kLaunch, kTickets, kCluster };
// NH: columns the softmax and fold threads work on, the q heads of a kv head (at most 8 per launch) -- not a runtime bound,
// which would put a branch in front of every column of the unrolled loops.  Instantiated for 4, 6, 7 and 8; other groups take the
// next wider one.  One kv head with 4 / 5 / 6 / 7 / 8 q heads, us a layer: 4.1 / 4.35 / 4.35 / 4.35 / 4.6 at 60 rows, 5.85 / 6.15 / 5.9 / 6.3 / 6.4
// at 8000, 6.9 / 7.3 / 7.4 / 7.5 / 7.7 at 32767: a group of 5 loses nothing by its dead column.
template <int NWG, int NS, int NH, bool APPEND, TcFold FOLD>
__global__ void __launch_bounds__((4 * NWG + 9) * 32, 1)
decodeI8TcKernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                 const __grid_constant__ CUtensorMap tmKn, const __grid_constant__ CUtensorMap tmVn,
                 const DecodeTcParams p) {
    using L = DecodeTcSmem<NWG, NS>;
    constexpr uint32_t kWG = NWG, kSoftThreads = 128u * NWG, kAllBar = NWG + 1u, kEndBar = NWG + 2u, kIssuedBar = NWG + 3u;
    constexpr uint32_t kFoldWarp0 = 4u * NWG, kProducerWarp = 4u * NWG + 4u, kMmaWarp0 = 4u * NWG + 5u;
    constexpr uint32_t kEndThreads = 32u * kProducerWarp;   // softmax + fold threads
    constexpr uint32_t T = kTcTile;
    const uint32_t chunk = blockIdx.x, kvHead = blockIdx.y, b = blockIdx.z;
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;

    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kBars);
    uint64_t *fullBar = bars, *emptyBar = bars + NS, *sFull = bars + 2 * NS, *pFull = sFull + 2 * NWG,
             *oFull = pFull + 2 * NWG, *oFree = oFull + 2 * NWG, *qFull = oFree + 2 * NWG, *rowFull = qFull + 1;
    uint32_t *tmemSlot = reinterpret_cast<uint32_t *>(smem + L::kTmemSlot);
    float *sHs = reinterpret_cast<float *>(smem + L::kHs);

    if (threadIdx.x == 0) {
        TC_STAMP(0);
        for (uint32_t s = 0; s < NS; ++s) {
            mbarInit(&fullBar[s], 1 + 32);
            mbarInit(&emptyBar[s], 1);
        }
        for (int i = 0; i < 2 * NWG; ++i) {
            mbarInit(&sFull[i], 1);
            mbarInit(&pFull[i], 4);  // (an arrival per warp: 128 of them serialise on the barrier)
            mbarInit(&oFull[i], 1);
            mbarInit(&oFree[i], 4);
        }
        mbarInit(qFull, 8);
        mbarInit(rowFull, 1);
        fenceBarrierInit();
        tmaPrefetchDesc(&tmK);
        tmaPrefetchDesc(&tmV);
    }
    // The length may live in device memory written by an earlier kernel; only a host-known
    // length lets the producer start before the dependency wait.
    uint32_t len = p.lenHost;
    const bool earlyOk = p.devLens == nullptr && p.devRowBase == nullptr && p.prefetchRows != 0;
    // a cluster shares the tiles that its sequence has, whatever the launch was sized for (a block may get none)
    auto tokensOfBlock = [&]() {
        return FOLD == TcFold::kCluster ? ((len + T - 1u) / T + gridDim.x - 1u) / gridDim.x * T : p.chunkTokens;
    };
    // inactive chunk (block-uniform): the merge derives the active count from len.  (The block that writes the output by
    // itself stays: a sequence without rows gets zeros.)
    auto inactive = [&]() { return FOLD != TcFold::kCluster && chunk * tokensOfBlock() >= len && (chunk != 0u || !p.directOut); };
    auto allocTmem = [&]() {
        if (warp != 0) return;
        __syncwarp();
        tmemAlloc(tmemSlot, L::kTmemCols);
        tmemRelinquish();
        tcFenceBefore();
    };
    // Tensor memory ahead of the dependency wait, where the length already says that the block will need it.
    const bool allocEarly = p.devLens == nullptr && !inactive();
    if (allocEarly) allocTmem();
    __syncthreads();
    if (p.dependent) gridDepLaunch();  // the next grid (the merge) may be scheduled as soon as room frees up

    if (!earlyOk) {
        // pulling this block's rows into L2 is right at any time: a row that a kernel in flight writes is read after the wait
        if (p.devLens == nullptr && p.devRowBase == nullptr && warp == kProducerWarp && lane < NS) {
            const uint32_t tok = chunk * tokensOfBlock() + lane * T, end = min(len, (chunk + 1u) * tokensOfBlock());
            if (tok < end) {
                const int row = static_cast<int>(static_cast<uint64_t>(b) * p.rowsPerSeq + tok);
                tmaPrefetchL2_3D(&tmK, 0, kvHead, row);
                tmaPrefetchL2_3D(&tmV, 0, kvHead, row);
            }
        }
        gridDepWait();
        if (p.devLens) len = min(p.devLens[b] + p.lenAdd, p.lenHost);  // (the host's length is the upper bound)
    }
    const uint32_t share = tokensOfBlock();
    const uint32_t t0 = chunk * share;
    if (inactive()) return;
    const uint32_t t1 = min(len, t0 + share);
    const uint32_t nTiles = t0 >= len ? 0u : (t1 - t0 + T - 1) / T;
    // Plain stream order: the kernels ahead are complete by now, and the block that stores a token's row lets the next grid
    // start behind that store (a call with TC_DECODE_PDL may request the row early).
    const bool storesRow = APPEND && p.appendK != nullptr && t1 == len && nTiles != 0u;
    if (!p.dependent && !storesRow) gridDepLaunch();
    constexpr bool CLUSTER = FOLD == TcFold::kCluster;
    __shared__ FoldInbox<CLUSTER ? 32 : 1> inbox;
    const uint32_t foldTotal = min(8u, p.group - p.colBase) * 32u;  // float4s of the outputs, and a block's share of them
    const uint32_t foldPer = CLUSTER ? (foldTotal + clusterSize() - 1u) / clusterSize() : 0u;
    if constexpr (CLUSTER) clusterHello();
    const uint64_t rowBase = p.devRowBase ? p.devRowBase[b] : static_cast<uint64_t>(b) * p.rowsPerSeq;
    if (!allocEarly) {
        allocTmem();
        __syncthreads();
    }
    tcFenceAfter();
    const uint32_t tmemBase = *reinterpret_cast<volatile uint32_t *>(tmemSlot);
    if (threadIdx.x == 0) TC_STAMP(1);
    // S of (warpgroup w, buffer bb) at columns 32 (2w + bb); O of the same pair 64 NWG columns further on

    if (warp == kProducerWarp) {
        // ------------------------------ TMA producer ------------------------------
        const uint64_t polFirst = l2PolicyEvictFirst(), polLast = l2PolicyEvictLast();
        auto prefetchNextPools = [&]() {
            // The same rows of the next call's pools into L2 (that call's TMA loads then hit L2).  The first NS tiles it requests
            // itself while it still waits for its q; what it waits for later are the tiles behind that ring.  So a block with more
            // tiles than the ring pulls those first (two at most, the more of the ring the fewer there are) and leaves HBM to
            // the rest.  28 / 4 heads, per layer, all tiles -> these: 32768 rows (7 tiles a block) 11.3 -> 10.7 us, 37000 (8)
            // 12.5 -> 11.7, 4 sequences of 8192 (8) 13.4 -> 12.7, 8 of 4400 (9) 11.9 -> 10.4, 2 of 22000 (10) 14.0 -> 13.0.
            const uint32_t first = nTiles > NS ? min(static_cast<uint32_t>(NS), 2u * (nTiles - NS) + 1u) : 0u;
            for (uint32_t it = first; it < min(nTiles, nTiles > kLateTiles ? NS + 4u : NS + 2u); ++it) {
                const int row = static_cast<int>(rowBase + t0 + it * T);
                if (p.l2Hints & 2) {
                    tmaPrefetchL2_3DHint(&tmKn, 0, kvHead, row, polLast);
                    tmaPrefetchL2_3DHint(&tmVn, 0, kvHead, row, polLast);
                } else {
                    tmaPrefetchL2_3D(&tmKn, 0, kvHead, row);
                    tmaPrefetchL2_3D(&tmVn, 0, kvHead, row);
                }
            }
        };
        if (APPEND && storesRow && lane < 8u) {
            // the rows this block will append, towards L2 (their final contents arrive there too)
            const char *src = reinterpret_cast<const char *>((lane < 4u ? p.appendK : p.appendV) +
                                                             (static_cast<size_t>(b) * p.nKV + kvHead) * 128u) + (lane & 3u) * 128u;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(src));
        }
        bool waited = !earlyOk;
        // K and V of tile `it`, completion on `bar` (its stage's fullBar, but for the tile with the appended row)
        auto requestRows = [&](uint32_t it, uint64_t *bar) -> bool {
            const uint32_t s = it % NS;
            if (it >= NS && !mbarWait<true>(&emptyBar[s], ((it / NS) - 1u) & 1u, p.err, kDevErrEmptyWait)) return false;
            const uint32_t tok = t0 + it * T;
            if (!waited && (tok + T > p.prefetchRows || it >= p.earlyStages)) {
                // rows the kernel in front may still be writing, or further ahead of the dependency
                // than the caller allows
                gridDepWait();
                waited = true;
            }
            uint8_t *st = smem + s * L::kStageBytes;
            const uint64_t row = rowBase + tok;
            if (lane == 0) {
                mbarExpectTx(bar, 2 * L::kTileBytes);
                if (p.l2Hints & 1) {
                    tmaLoad3DHint(st, &tmK, bar, 0, kvHead, static_cast<int>(row), polFirst);
                    tmaLoad3DHint(st + L::kTileBytes, &tmV, bar, 0, kvHead, static_cast<int>(row), polFirst);
                } else {
                    tmaLoad3D(st, &tmK, bar, 0, kvHead, static_cast<int>(row));
                    tmaLoad3D(st + L::kTileBytes, &tmV, bar, 0, kvHead, static_cast<int>(row));
                }
                if (it == 0) TC_STAMP(13);
                TC_STAMP(14);
            }
            return true;
        };
        // its row scales but that of row `skip` of the tile (T: all of them)
        auto requestScales = [&](uint32_t it, uint32_t skip) {
            const uint32_t s = it % NS;
            const uint64_t row = rowBase + t0 + it * T;
            float *sK = reinterpret_cast<float *>(smem + s * L::kStageBytes + 2 * L::kTileBytes);
            float *sV = sK + T;
#pragma unroll
            for (uint32_t idx = lane; idx < T; idx += 32) {
                uint64_t r = row + idx;
                r = r < p.totalRows ? r : p.totalRows - 1;
                if (APPEND && idx == skip) continue;
                cpAsync4(&sK[idx], p.ks + r * p.nKV + kvHead);
                cpAsync4(&sV[idx], p.vs + r * p.nKV + kvHead);
            }
            cpAsyncMbarArriveNoinc(&fullBar[s]);
        };
        // The tile that holds the row of a token being appended (the last tile of the sequence's last chunk) is requested apart
        // from the others.  The row goes into the tile itself behind the tile's copies, and into the pool: read back from
        // there, the tile came 1 us behind the other blocks' (28 / 4 heads, 4098 rows, f32 + int8: 6.75 us a layer, 6.5 like
        // this).  (All rows of the ring ahead of the first scales: these arrive behind 200 KB, 32768 rows 10.0 -> 11.6 us.)
        const uint32_t nLoop = storesRow ? nTiles - 1u : nTiles;
        bool okP = true;
        for (uint32_t it = 0; okP && it < nLoop; ++it) {
            okP = requestRows(it, &fullBar[it % NS]);
            if (okP) requestScales(it, T);
        }
        if (APPEND && storesRow && okP) {
            if (!waited) {
                gridDepWait();
                waited = true;
            }
            const uint64_t row = rowBase + (p.devLens ? p.devLens[b] + p.lenAdd : len) - 1u;
            // a length read from device memory is checked where it is known: outside the pool the
            // store is skipped and the error word says so
            const bool outside = row >= p.totalRows;
            if (outside && lane == 0) atomicOr(p.err, kDevErrRowBound);
            // (a device length above the host's bound: the row is stored, and lies behind the attended ones)
            const bool intoTile = !outside && row == rowBase + len - 1u;
            const uint32_t it = nTiles - 1u, inTile = len - 1u - (t0 + it * T);
            NewQuantRow<128, 128> fresh;
            const size_t src = (static_cast<size_t>(b) * p.nKV + kvHead) * 128u;
            fresh.load(p.appendK + src, p.appendV + src, lane);
            okP = requestRows(it, rowFull);
            if (okP) requestScales(it, intoTile ? inTile : T);
            okP = okP && mbarWait<true>(rowFull, 0, p.err, kDevErrFullWait);
            if (okP && !outside) {
                const uint64_t dst = row * p.nKV + kvHead;
                float4 *mk = nullptr, *mv = nullptr;
                if (p.mirK != nullptr) mk = reinterpret_cast<float4 *>(p.mirK) + dst * 32u, mv = reinterpret_cast<float4 *>(p.mirV) + dst * 32u;
                uint8_t *st = smem + (it % NS) * L::kStageBytes;
                float *sc = reinterpret_cast<float *>(st + 2 * L::kTileBytes);
                fresh.store(reinterpret_cast<uint32_t *>(p.k8w) + dst * 32u, reinterpret_cast<uint32_t *>(p.v8w) + dst * 32u,
                            const_cast<float *>(p.ks) + dst, const_cast<float *>(p.vs) + dst, mk, mv, intoTile ? st : nullptr,
                            st + L::kTileBytes, sc, sc + T, inTile, lane);
            }
            fenceProxyAsync();
            __syncwarp();
            if (okP && lane == 0) mbarArrive(&fullBar[it % NS]);
            // (the pool's row is next read by another launch's copies)
            asm volatile("fence.proxy.async.global;" ::: "memory");
            if (!p.dependent) {
                __threadfence();
                __syncwarp();
                gridDepLaunch();
            }
        }
        // all tiles of this block are requested: the next call's rows follow them into L2 (requested
        // earlier they sit in front of this block's own tiles in the queue: 10.2 against 9.1 us)
        // -- and a block of many tiles waits until its last one is in: HBM is what bounds it, and would be idle from there to the
        // next call's first requests, some 3 us.  That is room for four tiles a block.  Requested with its own last ring they
        // held that up by as much as they gained.  28 / 4 heads, per layer of calls above 48 MB, none -> four tiles behind the last, two / four / eight
        // layers of pools in turn, dependent launches: 8 sequences of 8192 rows (16 tiles a block) 14.1 / 14.2 / 14.5 -> 13.3 / 13.9 / 14.3 us, 16 of 4000
        // 13.5 / 14.1 / 14.5 -> 12.8 / 13.4 / 14.05, 2 of 30000 13.4 / 14.1 / 14.6 -> 12.9 / 13.3 / 13.9, 1 of 80000 16.9 / 17.6 / 17.9 -> 16.1 / 16.9 / 17.5; in
        // plain stream order 1 - 3 % of two and 2 - 4 % of eight layers, while four (L2 twice over) lose 2 - 5 %.  Eight layers of 8 x 8192 with
        // their session around them: 117.5 -> 116.4 us.  In blocks of fewer tiles, bound by latency, what comes
        // late comes too late: 2 of 22000 (10 tiles) 91.9 -> 95.1, 8 of 6000 (12 tiles) 87.5 -> 88.2.
        if (p.prefetchNext == 1 || (p.prefetchNext != 0 && nTiles > kLateTiles)) {
            const uint32_t last = nTiles - 1u;
            const bool in = nTiles <= kLateTiles || (okP && mbarWait(&fullBar[last % NS], (last / NS) & 1u, p.err, kDevErrFullWait));
            if (in && lane == 0) prefetchNextPools();
        }
    } else if (warp > kProducerWarp) {
        // -------------------------------- MMA issuers --------------------------------
        // Four issuing warps, so that no wait stands in front of another tile's products: score products and P.V products of
        // the even (warpgroup 0) and of the odd (warpgroup 1) tiles.  Warp-uniform control flow; the elected thread
        // executes the tcgen05 instructions.
        const uint32_t par = (warp - kMmaWarp0) & 1u;       // which tiles: j = par, par + 2, ...
        const bool pvRole = warp >= kMmaWarp0 + 2u;
        if (!pvRole) {
            constexpr uint32_t idQK = tcIdescI8(128, 32, 0, 0, 1, 1);   // K-major A (K tile), K-major B (q digits)
            const uint64_t dQd = tcDesc(smemAddr(smem + L::kQd), 16, 1024, 2);
            bool ok = mbarWait<true>(qFull, 0, p.err, kDevErrFullWait);
            if (lane == 0 && par == 0) TC_STAMP(15);
            for (uint32_t j = par; ok && j < nTiles; j += 2u) {
                const uint32_t s = j % NS, w = j % kWG, bb = (j / kWG) & 1u;
                // the P.V product of the buffers' previous tile (j - 2 NWG) is done: its scores have been read and its P tile
                // is free -- the softmax threads need not wait for that once more
                if (j >= 2u * kWG)
                    ok = mbarWait<true>(&oFull[2u * w + bb], ((j - 2u * kWG) / (2u * kWG)) & 1u, p.err, kDevErrMmaWait);
                ok = ok && mbarWait<true>(&fullBar[s], (j / NS) & 1u, p.err, kDevErrFullWait);
                if (lane == 0 && j < 8u) TC_STAMP(20 + j);
                if (!ok) break;
                tcFenceAfter();
                const uint64_t dK = tcDesc(smemAddr(smem + s * L::kStageBytes), 16, 1024, 2);
                const uint32_t tS = tmemBase + 32u * (2u * w + bb);
                if (electOne()) {
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k)  // 32 dims per instruction = 32 bytes inside the swizzle span
                        tcMmaI8(tS, dK + ((k * 32u) >> 4), dQd + ((k * 32u) >> 4), idQK, k > 0 ? 1u : 0u);
                    umaCommit(&sFull[2u * w + bb]);
                }
                __syncwarp();
            }
        } else {
            constexpr uint32_t idPV = tcIdescI8(128, 32, 1, 1, 1, 0);   // MN-major A (V tile), MN-major unsigned B (p digits)
            bool ok = true;
            for (uint32_t j = par; ok && j < nTiles; j += 2u) {
                const uint32_t s = j % NS, w = j % kWG, bb = (j / kWG) & 1u;
                // P of tile j published
                ok = mbarWait<true>(&pFull[2u * w + bb], (j / (2u * kWG)) & 1u, p.err, kDevErrMmaWait);
                // and the fold warpgroup has read the O buffer's previous contents (tile j - 2 NWG)
                if (ok && j >= 2u * kWG)
                    ok = mbarWait<true>(&oFree[2u * w + bb], ((j - 2u * kWG) / (2u * kWG)) & 1u, p.err, kDevErrMmaWait);
                if (!ok) break;
                tcFenceAfter();
                const uint64_t dV = tcDesc(smemAddr(smem + s * L::kStageBytes + L::kTileBytes), 16, 1024, 2);
                const uint64_t dP = tcDesc(smemAddr(smem + L::kP + (2u * w + bb) * 4096u), 16, 256, 6);
                const uint32_t tO = tmemBase + 64u * kWG + 32u * (2u * w + bb);
                if (electOne()) {
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k)  // 32 tokens per instruction: 4096 B of V, 1024 B of P
                        tcMmaI8(tO, dV + ((k * 4096u) >> 4), dP + ((k * 1024u) >> 4), idPV, k > 0 ? 1u : 0u);
                    umaCommit(&oFull[2u * w + bb]);
                    // K and V of the stage are consumed once these products are done (the score product
                    // of the tile completed before its P could be written)
                    umaCommit(&emptyBar[s]);
                }
                __syncwarp();
                if (lane == 0) TC_STAMP(16);
            }
        }
        // this warp issues nothing into tensor memory any more, whatever waits ran out: its owner may give it back
        namedBarArrive(kIssuedBar, 160);
    } else if (warp >= kFoldWarp0) {
        // ------------------------------ fold warpgroup ------------------------------
        // thread = one head dimension: takes every tile's integer P.V out of TMEM in tile order and
        // folds it into one f32 accumulator per head and softmax warpgroup, against that warpgroup's reference point
        // (a tile arrives with its fixed-point scale and, when it moved, the reference it was exponentiated against)
        const uint32_t wq = warp & 3u;
        const uint32_t row = wq * 32u + lane;
        const uint32_t laneBase = (wq * 32u) << 16;
        const float *meta = reinterpret_cast<const float *>(smem + L::kMeta);
        // accumulators and their reference points by softmax warpgroup: within one, the reference moves with a tile or two
        // of a call, and only then the accumulators are rescaled
        float oW[NWG][NH], M[NWG][NH];
#pragma unroll
        for (int w = 0; w < NWG; ++w)
#pragma unroll
            for (int h = 0; h < NH; ++h) oW[w][h] = 0.0f, M[w][h] = kNegBig;
        bool ok = true;
        for (uint32_t j0 = 0; ok && j0 < nTiles; j0 += kWG) {
#pragma unroll
            for (uint32_t w = 0; w < kWG; ++w) {
                const uint32_t j = j0 + w, bb = (j / kWG) & 1u, par = (j / (2u * kWG)) & 1u;
                if (j >= nTiles) break;
                ok = mbarWait<true>(&oFull[2u * w + bb], par, p.err, kDevErrMmaWait);
                if (!ok) break;
                tcFenceAfter();
                uint32_t r[32];
                tmemLd32(tmemBase + 64u * kWG + 32u * (2u * w + bb) + laneBase, r);
                const float *mt = meta + (4u * w + ((j / kWG) & 3u)) * 12u;
                const float2 em = *reinterpret_cast<const float2 *>(mt + 8);  // scale of the tile, whether the reference moved
                if (em.y != 0.0f) {
#pragma unroll
                    for (int h = 0; h < NH; ++h) {
                        const float mn = mt[h];  // (a reference only ever grows)
                        oW[w][h] *= fastExp2(M[w][h] - mn);
                        M[w][h] = mn;
                    }
                }
                tmemLdWait();
                tcFenceBefore();
                __syncwarp();
                if (lane == 0) mbarArrive(&oFree[2u * w + bb]);   // the buffer and its meta slot may be reused
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    // column 4h + i carries byte i of the fixed-point probability: weight 256^i; a sum is below 2^22, so
                    // two of them combine exactly in 32 bits
                    const int lo = static_cast<int>(r[4 * h + 1]) * 256 + static_cast<int>(r[4 * h]);
                    const int hi = static_cast<int>(r[4 * h + 3]) * 256 + static_cast<int>(r[4 * h + 2]);
                    const float c = fmaf(__int2float_rn(hi), 65536.0f, __int2float_rn(lo));
                    oW[w][h] = fmaf(c, em.x, oW[w][h]);
                }
                if (threadIdx.x == kFoldWarp0 * 32u && j + 1u == nTiles) TC_STAMP(10);
            }
        }
        float o[8], Mx[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            o[h] = 0.0f, Mx[h] = kNegBig;
            if (h < NH) {
#pragma unroll
                for (int w = 0; w < NWG; ++w) Mx[h] = fmaxf(Mx[h], M[w][h]);
#pragma unroll
                for (int w = 0; w < NWG; ++w) o[h] = fmaf(oW[w][h], fastExp2(M[w][h] - Mx[h]), o[h]);
            }
        }
        // every P tile has been consumed (its O was waited for above): their space is the scratch
        float *scr = reinterpret_cast<float *>(smem + L::kP);
        namedBarSync(kEndBar, kEndThreads);
#pragma unroll
        for (int h = 0; h < 8; ++h) scr[h * 128u + row] = o[h];
        if (threadIdx.x == kFoldWarp0 * 32u) {
#pragma unroll
            for (int h = 0; h < 8; ++h) scr[8 * 128 + h] = Mx[h];
        }
        namedBarSync(kEndBar, kEndThreads);
    } else {
        // ---------------------------- softmax warpgroups ----------------------------
        const uint32_t w = warp >> 2;                       // warpgroup: tiles j = w, w + NWG, ...
        const uint32_t wq = warp & 3u;                      // TMEM lane quarter of this warp
        const uint32_t row = wq * 32u + lane;               // token of the tile
        const uint32_t laneBase = (wq * 32u) << 16;
        const uint32_t wgBar = 1u + w;                      // named barrier of the warpgroup
        float *red = reinterpret_cast<float *>(smem + L::kRed) + w * 48u;
        float *meta = reinterpret_cast<float *>(smem + L::kMeta);

        // pull q towards L2 while waiting (harmless if the kernel in front is still writing it)
        if (lane == 0 && warp < 8u && p.colBase + warp < p.group)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.q + (static_cast<size_t>(b) * p.nHeads + kvHead * p.group + p.colBase + warp) * 128u));
        gridDepWait();  // q comes from a kernel that may still be running
        if (threadIdx.x == 0) TC_STAMP(2);
        // ---- q of head `warp` of this kv head -> three signed base-128 digit planes ----
        if (warp < 8u) {
            const uint32_t h = warp;  // 8 softmax warps = the 8 MMA columns
            const bool valid = p.colBase + h < p.group;
            const float4 qv = valid ? __ldg(reinterpret_cast<const float4 *>(
                                              p.q + (static_cast<size_t>(b) * p.nHeads + kvHead * p.group + p.colBase + h) * 128u) + lane)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
            float amax = fmaxf(fmaxf(fabsf(qv.x), fabsf(qv.y)), fmaxf(fabsf(qv.z), fabsf(qv.w)));
#pragma unroll
            for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            // |q| * 2^-e < 1 with e = floor(log2 amax) + 1; digits of X = rint(q * 2^(20 - e)), |X| <= 2^20
            int e = static_cast<int>((__float_as_uint(amax) >> 23) & 0xffu) - 126;
            e = amax > 0.0f ? max(-100, min(100, e)) : 0;
            const float toFix = __uint_as_float(static_cast<uint32_t>(127 + 20 - e) << 23);
            auto digits = [&](float x, int &d0, int &d1, int &d2) {
                const int X = __float2int_rn(x * toFix);
                d2 = ((X + 64) & 127) - 64;
                const int X1 = (X - d2) >> 7;
                d1 = ((X1 + 64) & 127) - 64;
                d0 = (X1 - d1) >> 7;
            };
            int d0[4], d1[4], d2[4];
            digits(qv.x, d0[0], d1[0], d2[0]);
            digits(qv.y, d0[1], d1[1], d2[1]);
            digits(qv.z, d0[2], d1[2], d2[2]);
            digits(qv.w, d0[3], d1[3], d2[3]);
            auto pack = [](const int (&d)[4]) {
                return (static_cast<uint32_t>(d[0]) & 0xffu) | ((static_cast<uint32_t>(d[1]) & 0xffu) << 8) |
                       ((static_cast<uint32_t>(d[2]) & 0xffu) << 16) | ((static_cast<uint32_t>(d[3]) & 0xffu) << 24);
            };
            // row n = plane * 8 + head, 128 bytes of dims, 16-byte units xor-swizzled by the row (128-byte swizzle)
            uint8_t *qd = smem + L::kQd;
            const uint32_t unit = lane >> 2, inUnit = (lane & 3u) * 4u;
            auto put = [&](uint32_t n, uint32_t word) {
                *reinterpret_cast<uint32_t *>(qd + n * 128u + ((unit ^ (n & 7u)) << 4) + inUnit) = word;
            };
            put(h, pack(d0));
            put(8u + h, pack(d1));
            put(16u + h, pack(d2));
            put(24u + h, 0u);
            // log2-domain scale of this head's integer scores: invSqrt * log2(e) * 2^(e - 20)
            if (lane == 0)
                sHs[h] = valid ? p.invSqrt * kLog2e * __uint_as_float(static_cast<uint32_t>(127 + e - 20) << 23) : 0.0f;
            fenceProxyAsync();
            __syncwarp();
            if (lane == 0) mbarArrive(qFull);
        }
        if (threadIdx.x == 0) TC_STAMP(3);
        namedBarSync(kAllBar, kSoftThreads);  // head scales visible to every warpgroup
        float hs[NH];
#pragma unroll
        for (int h = 0; h < NH; ++h) hs[h] = sHs[h];

        float mref[NH], l[NH];
#pragma unroll
        for (int h = 0; h < NH; ++h) mref[h] = kNegBig, l[h] = 0.0f;
        float Eref = 0.0f, invW = 0.0f;  // power of two above every V scale seen; 2^24 / Eref
        bool ok = true;

        for (uint32_t j = w; j < nTiles; j += kWG) {
            const uint32_t s = j % NS, bb = (j / kWG) & 1u;
            // ---- this thread's token against the NH columns ----
            if (!mbarWait<true>(&sFull[2u * w + bb], (j / (2u * kWG)) & 1u, p.err, kDevErrMmaWait)) {
                ok = false;
                break;
            }
            tcFenceAfter();
            if (threadIdx.x == 0 && j == 0) TC_STAMP(4);
            uint32_t ra[16], rb[8];
            const uint32_t tS = tmemBase + 32u * (2u * w + bb) + laneBase;
            tmemLd16(tS, ra);
            tmemLd8(tS + 16u, rb);
            const float *sK = reinterpret_cast<const float *>(smem + s * L::kStageBytes + 2 * L::kTileBytes);
            const bool valid = t0 + j * T + row < t1;
            const float skr = sK[row];
            const float svr = valid ? sK[T + row] : 0.0f;
            tmemLdWait();
            // x = score - reference point (log2 units)
            float f[NH], x[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                // digit planes 1 and 2 combine exactly in 32 bits (below 2^20 each)
                const int lo = static_cast<int>(ra[8 + h]) * 128 + static_cast<int>(rb[h]);
                f[h] = fmaf(i2f(ra[h]), 16384.0f, __int2float_rn(lo));
                x[h] = fmaf(f[h], skr * hs[h], -mref[h]);
            }
            if (t0 + (j + 1u) * T > t1) {  // the last tile: rows behind the range (whatever their scales hold)
#pragma unroll
                for (int h = 0; h < NH; ++h) x[h] = valid ? x[h] : -INFINITY;
            }
            float top = x[0];
#pragma unroll
            for (int h = 1; h < NH; ++h) top = fmaxf(top, x[h]);
            // (the first tile of a warpgroup always moves it)
            const bool moved = j == w || barOr(wgBar, 128, svr >= Eref || top > kTcLazyLog2);
            if (moved) {
                // rare: the reference point of a head (or the bound of the V scales) has to move --
                // tile maxima over the warpgroup, then every thread applies the same update
                float tm[NH + 1];
#pragma unroll
                for (int h = 0; h < NH; ++h) x[h] = tm[h] = valid ? f[h] * (skr * hs[h]) : -INFINITY;
                tm[NH] = svr;
#pragma unroll
                for (int i = 0; i <= NH; ++i) tm[i] = warpMax(tm[i]);
                if (lane == 0) {
#pragma unroll
                    for (int i = 0; i <= NH; ++i) red[wq * 12u + i] = tm[i];
                }
                namedBarSync(wgBar, 128);  // (the next vote lies between these reads and the next rare pass's writes)
#pragma unroll
                for (int i = 0; i <= NH; ++i) tm[i] = fmaxf(fmaxf(red[i], red[12 + i]), fmaxf(red[24 + i], red[36 + i]));
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    const float mn = fmaxf(mref[h], tm[h]);
                    l[h] *= fastExp2(mref[h] - mn);
                    mref[h] = mn;
                    x[h] -= mn;
                }
                if (tm[NH] >= Eref) {
                    uint32_t eb = (__float_as_uint(tm[NH]) & 0x7f800000u) + 0x00800000u;  // 2^(floor(log2) + 1)
                    eb = min(max(eb, 24u << 23), 253u << 23);
                    Eref = __uint_as_float(eb);
                    invW = __uint_as_float((127u + 24u + 127u) * (1u << 23) - eb);  // 2^24 / Eref
                }
            }
            // p, l, and p * sv as 32-bit fixed point (8.24 against Eref): its bytes are the digit planes
            const float wv = svr * invW;
            uint32_t X[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                X[h] = 0u;
                if (h < NH) {
                    const float pr = fastExp2(x[h < NH ? h : 0]);
                    l[h < NH ? h : 0] += pr;
                    X[h] = __float2uint_rn(pr * wv);
                }
            }
            uint8_t *pt = smem + L::kP + (2u * w + bb) * 4096u + row * 32u;
            const uint32_t sw = (row >> 2) & 1u;  // 32-byte swizzle: 16-byte halves swap on rows 4..7 of every 8
            *reinterpret_cast<uint4 *>(pt + ((0u ^ sw) << 4)) = make_uint4(X[0], X[1], X[2], X[3]);
            *reinterpret_cast<uint4 *>(pt + ((1u ^ sw) << 4)) = make_uint4(X[4], X[5], X[6], X[7]);
            if (row == 0) {
                // what the fold warpgroup needs with this tile: the scale of its fixed-point probabilities and, when they
                // moved, the reference points these were taken against
                float *mt = meta + (4u * w + ((j / kWG) & 3u)) * 12u;
                if (moved) {
#pragma unroll
                    for (int h = 0; h < NH; ++h) mt[h] = mref[h];
                }
                *reinterpret_cast<float2 *>(mt + 8) = make_float2(Eref * 5.9604644775390625e-8f, moved ? 1.0f : 0.0f);  // Eref * 2^-24
            }
            fenceProxyAsync();
            tcFenceBefore();
            __syncwarp();
            if (lane == 0) mbarArrive(&pFull[2u * w + bb]);
            if (threadIdx.x == 0 && j / kWG < 4u) TC_STAMP(5 + j / kWG);
        }

        // ---- row sums of this warpgroup, then the end of the block ----
#pragma unroll
        for (int h = 0; h < NH; ++h)
#pragma unroll
            for (int off = 16; off; off >>= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], off);
        float *scr = reinterpret_cast<float *>(smem + L::kP);
        float *oS = scr;                          // [8][128] from the fold warpgroup, then its reference points [8]
        float *mF = scr + 8 * 128;
        float *mS = mF + 8;                       // [NWG][8]
        float *lS = mS + NWG * 8;                 // [4 NWG warps][8]
        namedBarSync(kEndBar, kEndThreads);       // the fold warpgroup is through: every P tile has been consumed
        if (lane == 0) {
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                lS[warp * 8u + h] = l[h];
                if (wq == 0) mS[w * 8u + h] = mref[h];
            }
        }
        namedBarSync(kEndBar, kEndThreads);
        if (threadIdx.x == 0) TC_STAMP(11);
        if constexpr (CLUSTER) clusterHelloWait();
        if (warp < 8u) {
            const uint32_t tid = threadIdx.x;  // 0..255: head tid / 32, dims 4 (tid % 32) ..
            const uint32_t h = tid >> 5, d4 = tid & 31u;
            if (p.colBase + h < p.group) {
                // the accumulator is relative to the fold warpgroup's reference point, which is the
                // largest of the warpgroups' (a reference only ever grows)
                const float M = mF[h];
                const float4 acc = *reinterpret_cast<const float4 *>(oS + h * 128u + 4u * d4);
                float lsum = 0.0f;
#pragma unroll
                for (int g = 0; g < NWG; ++g) {
                    const float a = fastExp2(mS[g * 8 + h] - M);   // a warpgroup without tiles: exp2(-1e30) = 0
                    const float lg = (lS[(4 * g) * 8 + h] + lS[(4 * g + 1) * 8 + h]) +
                                     (lS[(4 * g + 2) * 8 + h] + lS[(4 * g + 3) * 8 + h]);
                    lsum = fmaf(a, lg, lsum);
                }
                const size_t oidx = static_cast<size_t>(b) * p.nHeads + kvHead * p.group + p.colBase + h;
                if constexpr (CLUSTER) {
                    inboxPush<32>(inbox, tid, foldPer, clusterRank(), M, lsum, acc);
                } else if (p.directOut) {
                    const float inv = lsum > 0.0f ? 1.0f / lsum : 0.0f;
                    *reinterpret_cast<float4 *>(p.out + oidx * 128u + 4u * d4) =
                            make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
                } else {
                    const size_t pidx = oidx * p.numChunks + chunk;
                    *reinterpret_cast<float4 *>(p.pAcc + pidx * 128u + 4u * d4) = acc;
                    if (d4 == 0) {
                        // natural-log units: the merge contract is w = exp2((m - M) * log2e)
                        p.pM[pidx] = M > -1e29f ? M * 0.6931471805599453f : kNegBig;
                        p.pL[pidx] = lsum;
                    }
                }
            }
        }
        if (FOLD == TcFold::kTickets && !p.directOut && p.tickets != nullptr) {
            // ---- merge inside the kernel: the block that arrives last at its (sequence, kv head)
            // counter folds all chunk partials of the kv head's q heads.  Nobody waits: every block
            // publishes its partial, takes a ticket and leaves unless the ticket is the last one.
            uint32_t *sTicket = reinterpret_cast<uint32_t *>(lS + 4 * NWG * 8);
            __threadfence();  // this thread's partial stores are visible device-wide before the ticket
            namedBarSync(kAllBar, kSoftThreads);
            uint32_t *ctr = p.tickets + static_cast<size_t>(b) * p.nKV + kvHead;
            if (threadIdx.x == 0) *sTicket = atomicAdd(ctr, 1u);
            namedBarSync(kAllBar, kSoftThreads);
            const uint32_t nActive = min((len + p.chunkTokens - 1u) / p.chunkTokens, gridDim.x);
            if (*sTicket == nActive - 1u) {
                __threadfence();
                if (threadIdx.x == 0) *ctr = 0u;  // ready for the next call on this stream
                const uint32_t h = warp;          // one warp per q head, lane = four dims
                if (warp < 8u && p.colBase + h < p.group) {
                    const size_t oidx = static_cast<size_t>(b) * p.nHeads + kvHead * p.group + p.colBase + h;
                    const float *gm = p.pM + oidx * p.numChunks, *gl = p.pL + oidx * p.numChunks;
                    const float *ga = p.pAcc + oidx * p.numChunks * 128u + 4u * lane;
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    float M = kNegBig, Lsum = 0.0f;
                    // chunk partials in groups of 32: lane c holds (m, l) of chunk c0 + c
                    for (uint32_t c0 = 0; c0 < nActive; c0 += 32u) {
                        const uint32_t c = c0 + lane;
                        const float lc = c < nActive ? __ldcg(gl + c) : 0.0f;
                        const float mc = (c < nActive && lc > 0.0f) ? __ldcg(gm + c) : kNegBig;
                        float gmx = mc;
#pragma unroll
                        for (int off = 16; off; off >>= 1) gmx = fmaxf(gmx, __shfl_xor_sync(0xffffffffu, gmx, off));
                        const float Mn = fmaxf(M, gmx);
                        const float sOld = fastExp2((M - Mn) * kLog2e);
                        acc.x *= sOld, acc.y *= sOld, acc.z *= sOld, acc.w *= sOld;
                        Lsum *= sOld;
                        M = Mn;
                        const float wc = lc > 0.0f ? fastExp2((mc - M) * kLog2e) : 0.0f;
                        float wl = wc * lc;
#pragma unroll
                        for (int off = 16; off; off >>= 1) wl += __shfl_xor_sync(0xffffffffu, wl, off);
                        Lsum += wl;
                        const uint32_t n = min(32u, nActive - c0);
#pragma unroll 8
                        for (uint32_t i = 0; i < n; ++i) {
                            const float wi = __shfl_sync(0xffffffffu, wc, i);
                            const float4 a = __ldcg(reinterpret_cast<const float4 *>(ga + static_cast<size_t>(c0 + i) * 128u));
                            acc.x = fmaf(wi, a.x, acc.x);
                            acc.y = fmaf(wi, a.y, acc.y);
                            acc.z = fmaf(wi, a.z, acc.z);
                            acc.w = fmaf(wi, a.w, acc.w);
                        }
                    }
                    const float inv = Lsum > 0.0f ? 1.0f / Lsum : 0.0f;
                    *reinterpret_cast<float4 *>(p.out + oidx * 128u + 4u * lane) =
                            make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
                }
            }
        }
    }
    if (threadIdx.x == 0) TC_STAMP(12);
    // (every read of tensor memory lies in front of the barrier that the fold and the softmax warps met at, and the issuing
    // warps are through -- long ago, and with every product waited for by the fold warps, unless a wait ran out)
    if (warp == 0) {
        namedBarSync(kIssuedBar, 160);
        tcFenceAfter();
        tmemDealloc(tmemBase, L::kTmemCols);
    }
    if constexpr (CLUSTER) {
        // every block's results are in the inboxes of the blocks that put them together
        if (warp >= kFoldWarp0) clusterHelloWait();
        clusterSync();
        const uint32_t idx = clusterRank() * foldPer + threadIdx.x;
        if (threadIdx.x < foldPer && idx < foldTotal) {
            float M, l;
            float4 acc;
            inboxTake<32>(inbox, threadIdx.x, foldPer, clusterSize(), M, l, acc);
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            const size_t oidx = static_cast<size_t>(b) * p.nHeads + kvHead * p.group + p.colBase + (idx >> 5);
            *reinterpret_cast<float4 *>(p.out + oidx * 128u + 4u * (idx & 31u)) =
                    make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
        }
    }
}

// Host side: arguments were validated by the caller (decodeI8Common in decode_i8.cu).
int decodeI8Tc(const tc_decode_i8_batch *d, uint32_t lenHost, uint32_t lenAdd, const F32Mirror &mir, cudaStream_t st) {
    const uint32_t hd = 128;
    const uint32_t group = d->nHeads / d->nKV;
    using Smem = DecodeTcSmem<2, 6>;
    // A cluster per (sequence, kv head) folds without partials and merge launch.  It is taken when all of them are resident
    // at once (16 blocks: 7, 8: 15, 4: 33, 2: 74, a block filling an SM) and their blocks, fewer than the merge form's, do not
    // cost more than the launch: a tile more per block takes 0.25 - 0.3 us while latency is what bounds it, and a fold over 16 blocks
    // more than one over 8.  So up to five tiles more per block for 16 of them and nine for fewer -- where the clusters keep 5 / 8 of the
    // SMs busy.  Where they do not, a tile is not latency alone, the rows come in over those SMs only: five for 8 blocks, three for 4 and 2.
    // Cluster against merge, 28 / 4 heads unless said, rows asked for early (TC_DECODE_PDL) / plain stream order, per layer, tiles a block in brackets:
    //   16 blocks: 1 sequence of 12708 - 19749 rows (3 -> 7, 5 -> 10) 0.70 - 0.96 / 0.72 - 1.015; of 30000 (7 -> 15) 1.04;
    //   8 blocks, 96 of them: 3 sequences of 10520 - 27057 (7 -> 11, 18 -> 27) 0.83 - 0.92 / 0.93 - 1.01;
    //   8 blocks, 64: 2 of 6357 - 9275 (3 -> 7, 5 -> 10) 0.88 - 0.92 / 0.93 - 0.99, of 15351 (7 -> 15) 1.06 / 1.06; 40 / 8, one of 11204 (5 -> 11) 1.045 / 1.08,
    //     of 15351 1.09 / 1.10;
    //   4 blocks, 96 and 112: 6 and 7 of 5262 - 23855 (7 -> 11, 38 -> 47) 0.81 - 0.96 / 0.91 - 1.0; 64: 4 of 5969 (6 -> 12) 1.11 / 1.14, of 7678 1.04 / 1.15;
    //     80: 5 of 4941 - 9275 (6 -> 10, 11 -> 19) 1.01 - 1.07 / 0.99 - 1.06;
    //   2 blocks, 96: 12 of 2632 - 6770 (7 -> 11, 18 -> 27) 0.88 - 0.96 / 0.95 - 1.01; 72: 12 / 2, 18 of 2320 - 4356 (5 -> 10, 9 -> 18) 1.03 - 1.08 / 1.07 - 1.09.
    // With ragged device lengths the cluster also shares every sequence evenly among its blocks, where the
    // merge form cuts chunks by the longest one.  There the line is 20 tiles per block of the longest sequence for 16 blocks: cluster
    // against merge, 2 / 3 / 4 / 8 sequences of up to 6000 rows (6 - 12 tiles) 0.44 / 0.48 / 0.66 / 0.67 of the time, up to 20000
    // (20 tiles, 2 and 3 sequences) 0.83 and 0.87, up to 32768 (32, 2 and 3) 1.15; and 26 for fewer: 2 and 3 of up to 26000 (26 tiles) 0.83 and 0.82,
    // 4 / 5 / 6 / 8 of up to 12000 (24) 0.92 / 0.94 / 0.96 / 0.97, 12 and 16 of up to 6000 (24) 0.91 and 0.92, 4 / 5 / 6 / 8 of up to 16000 (32) 1.19 / 1.19 / 1.09 / 1.05.
    static ClusterSetup setup;
    const uint32_t *limits = nullptr;
    int rc = setupCluster(setup, decodeI8TcKernel<2, 6, 8, true, TcFold::kCluster>, Smem::kThreads, Smem::kTotal, &limits);
    if (rc != TC_OK) return rc;
    DecodePlan pl = planDecode(d->batch, d->nKV, d->maxLen, d->numChunks, kTcTile, d->lens == nullptr, 1u);
    uint32_t cluster = 1;
    const bool partials = d->pAcc && d->pM && d->pL;  // (without them a merge is not to be had: nine for all)
    if (pl.chunksPerSeq > 1 && !d->partialsOnly && d->mergeTickets == nullptr) {
        const uint32_t tiles = (d->maxLen + kTcTile - 1) / kTcTile;
        for (uint32_t lg = 4; lg >= 1 && cluster == 1; --lg) {
            const uint32_t n = 1u << lg;
            const bool busy = n * d->nKV * d->batch * 8u >= static_cast<uint32_t>(numSMs()) * 5u;
            const uint32_t more = n == 16u ? 5u : (busy || !partials ? 9u : (n == 8u ? 5u : 3u));
            const uint32_t most = d->lens == nullptr || d->batch == 1 ? pl.chunkTokens / kTcTile + more : n == 16u ? 20u : 26u;  // tiles per block
            if (n / 2u >= tiles || limits[lg] < d->nKV * d->batch || (tiles + n - 1u) / n > most) continue;
            cluster = n;
            pl.chunksPerSeq = n;
        }
    }
    const bool pdl = (d->flags & TC_DECODE_PDL) != 0;
    const bool direct = (pl.chunksPerSeq == 1 || cluster > 1) && !d->partialsOnly;
    if (!direct) TC_REQUIRE(partials, TC_EWORKSPACE, "decode_i8: partial buffers are required");
    if (d->chunksUsed) *d->chunksUsed = cluster > 1 ? 1u : pl.chunksPerSeq;  // (a cluster's blocks write no slots)
    TC_REQUIRE(d->nKV <= 65535, TC_EUNSUPPORTED, "decode_i8: %u kv heads", d->nKV);

    TensorMapKey key;
    memset(&key, 0, sizeof(key));
    key.rank = 3;
    key.elemBytes = 1;
    key.swizzle = 3;
    key.dims[0] = hd;
    key.dims[1] = d->nKV;
    key.dims[2] = d->totalRows;
    key.strides[0] = hd;
    key.strides[1] = static_cast<uint64_t>(d->nKV) * hd;
    key.box[0] = 128;
    key.box[1] = 1;
    key.box[2] = kTcTile;
    CUtensorMap tmK, tmV;
    key.base = d->k8;
    rc = getTensorMap(key, &tmK);
    if (rc != TC_OK) return rc;
    key.base = d->v8;
    rc = getTensorMap(key, &tmV);
    if (rc != TC_OK) return rc;
    CUtensorMap tmKn = tmK, tmVn = tmV;
    // the next call's pools, pulled into L2 behind this call's rows; larger calls keep HBM busy by themselves.  (With the hint
    // against without it, per layer of pools that do not fit L2 together: 20000 rows 8.70 / 9.25 us, 32768 rows 10.90 /
    // 10.98, 47000 rows (46 MiB) 14.04 / 13.55, 50000 rows 14.25 / 14.02, 80000 rows 18.13 / 18.46; 4 sequences of 8192 rows
    // 12.2 / 11.7, 8 of 8192 14.24 / 14.60.  It pays where a call is short; from some 30 MB on it is within 4 % either way.)  Blocks of many tiles
    // pull them when their own are in (kLateTiles), which pays up to 80 MB: 2 sequences of 40000 rows (82 MB) 17.1 / 17.0 us a layer of eight,
    // 8 of 12000 (98 MB) 18.2 / 18.25.
    const uint64_t callBytes = static_cast<uint64_t>(d->batch) * d->maxLen * d->nKV * hd * 2ull;
    // (Between 48 and 80 MB a hint that a copy could not follow is no error: those calls used to go without one.)
    const bool nextAligned = ((reinterpret_cast<uintptr_t>(d->nextK8) | reinterpret_cast<uintptr_t>(d->nextV8)) & 15u) == 0;
    const int prefetchNext = d->nextK8 == nullptr || d->nextV8 == nullptr || callBytes > (80ull << 20) ? 0
                             : callBytes <= (48ull << 20)                                              ? 1
                                                                                                       : (nextAligned ? 2 : 0);
    if (prefetchNext) {
        TC_REQUIRE(nextAligned, TC_EINVAL, "decode_i8: nextK8/nextV8 need 16-byte alignment");
        key.base = d->nextK8;
        rc = getTensorMap(key, &tmKn);
        if (rc != TC_OK) return rc;
        key.base = d->nextV8;
        rc = getTensorMap(key, &tmVn);
        if (rc != TC_OK) return rc;
    }

    DecodeTcParams prm;
    prm.q = d->q;
    prm.out = d->out;
    prm.ks = d->ks;
    prm.vs = d->vs;
    prm.nextK8 = d->nextK8;
    prm.nextV8 = d->nextV8;
    prm.appendK = d->appendK;
    prm.appendV = d->appendV;
    prm.mirK = mir.k, prm.mirV = mir.v;
    prm.k8w = const_cast<int8_t *>(d->k8);
    prm.v8w = const_cast<int8_t *>(d->v8);
    prm.pAcc = d->pAcc;
    prm.pM = d->pM;
    prm.pL = d->pL;
    // the in-kernel merge serves one launch per call (q-head groups of at most 8) and needs the output
    const bool fused = d->mergeTickets != nullptr && !direct && !d->partialsOnly && group <= 8;
    prm.tickets = fused ? d->mergeTickets : nullptr;
    prm.devLens = d->lens;
    prm.devRowBase = d->rowBase;
    prm.rowsPerSeq = d->rowsPerSeq;
    prm.totalRows = d->totalRows;
    prm.lenHost = lenHost;
    prm.lenAdd = lenAdd;
    prm.nHeads = d->nHeads;
    prm.nKV = d->nKV;
    prm.group = group;
    prm.colBase = 0;
    prm.chunkTokens = pl.chunkTokens;
    prm.numChunks = d->numChunks;
    prm.prefetchRows = pdl ? d->prefetchRows : 0;
    prm.invSqrt = d->invSqrt;
    prm.directOut = direct ? 1 : 0;
    prm.dependent = pdl ? 1 : 0;
    prm.prefetchNext = prefetchNext;
    // Under programmatic dependent launch the producer requests a whole ring of old rows while the
    // kernels ahead drain (7B shape, 32768 rows, batch 1: 12.4 us per layer against 13.5 with one
    // stage).  The block's own tiles are read once (evict-first); the next call's rows pulled in
    // behind them are kept (evict-last) -- with plain policies the hint gained nothing.
    prm.earlyStages = 6;
    prm.l2Hints = 3;
    prm.err = devErrorWord();
    TC_REQUIRE(prm.err != nullptr, TC_ECUDA, "decode_i8: no device error word");
#ifdef TC_TRACE
    {
        extern unsigned long long *g_tcTrace;
        static unsigned callNo = 0;
        prm.trace = g_tcTrace ? g_tcTrace + static_cast<size_t>((callNo++) & 3u) * 160 * 32 : nullptr;
    }
#endif

    // (Four softmax warpgroups with a five-stage ring were measured and dropped: 11.5 against 8.3 us
    // per layer for the split launch alone at 32768 rows, 53.9 against 47.0 us at batch 8.)
    // (each way of coming together is an instantiation of its own for the same reason as the append)
    using Kern = decltype(&decodeI8TcKernel<2, 6, 8, true, TcFold::kLaunch>);
#define TC_KERNS(NH, APPEND) {decodeI8TcKernel<2, 6, NH, APPEND, TcFold::kLaunch>, decodeI8TcKernel<2, 6, NH, APPEND, TcFold::kCluster>}
    static const Kern kerns[4][2][2] = {{TC_KERNS(4, false), TC_KERNS(4, true)},
                                        {TC_KERNS(6, false), TC_KERNS(6, true)},
                                        {TC_KERNS(7, false), TC_KERNS(7, true)},
                                        {TC_KERNS(8, false), TC_KERNS(8, true)}};
#undef TC_KERNS
    static const Kern ticketKerns[2] = {decodeI8TcKernel<2, 6, 8, false, TcFold::kTickets>,
                                        decodeI8TcKernel<2, 6, 8, true, TcFold::kTickets>};
    static bool attrDone[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attrDone[dev]) {
        auto attributes = [](Kern k) {
            TC_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::kTotal));
            TC_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            return static_cast<int>(TC_OK);
        };
        for (auto &byHeads : kerns)
            for (auto &byAppend : byHeads)
                for (Kern k : byAppend)
                    if ((rc = attributes(k)) != TC_OK) return rc;
        for (Kern k : ticketKerns)
            if ((rc = attributes(k)) != TC_OK) return rc;
        attrDone[dev] = true;
    }
    const uint32_t append = d->appendK != nullptr ? 1 : 0, heads = group <= 4 ? 0 : group <= 6 ? 1 : group == 7 ? 2 : 3;
    const Kern kern = fused ? ticketKerns[append] : kerns[heads][append][cluster > 1 ? 1 : 0];
    // (without TC_DECODE_PDL prefetchRows is 0 and every block waits for the kernels ahead first thing)
    // a launch serves 8 q heads per kv head (the MMA columns); wider groups take one launch per
    // block of 8 and stream the rows again
    for (uint32_t cb = 0; cb < group; cb += 8) {
        prm.colBase = cb;
        rc = launchDependent(kern, dim3(pl.chunksPerSeq, d->nKV, d->batch), Smem::kThreads, Smem::kTotal, st, cluster, tmK,
                             tmV, tmKn, tmVn, prm);
        if (rc != TC_OK) return rc;
    }
    if (direct || d->partialsOnly || fused) return TC_OK;
    return launchMerge(d->pAcc, d->pM, d->pL, d->out, d->batch, d->nHeads, d->numChunks, pl.chunksPerSeq, hd, d->lens,
                       lenAdd, pl.chunkTokens, nullptr, pdl, st);
}

#ifdef TC_TRACE
unsigned long long *g_tcTrace = nullptr;
#endif

}  // namespace tc

#ifdef TC_TRACE
extern "C" void tc_debug_trace(unsigned long long *buf) { tc::g_tcTrace = buf; }
#endif
