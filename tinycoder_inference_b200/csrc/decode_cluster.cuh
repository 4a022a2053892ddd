// decode_cluster.cuh -- what the mma.sync decode kernels (f32, fp16 and head_dim-256 int8 stores) share
// around their inner loops: the split of a sequence over clusters of blocks, the fold of the partial
// results through distributed shared memory, and the new token's row and rotation.
//
// A block streams a token range of ONE kv head; the blocks of a cluster hold neighbouring ranges of the same
// kv head and fold their (m, l, acc) through each other's shared memory.  When one cluster covers the
// sequence the result goes straight to the output: no partials in global memory, no merge launch.  Longer
// sequences take blocks on their own and the merge (merge.cu).
//
// What bounds these kernels up to some ten thousand rows is the chain of launches and barriers, not the bytes: on
// B200 a launch that waits for the one in front of it costs 3.1 - 3.7 us in stream order, 2.0 us under programmatic
// dependent launch (0.8 in a graph).  Measured per layer in a graph, 28 q / 4 kv heads of 128, fp16: one block per
// kv head 5.7 us at 200 rows, two blocks and a merge 6.5, a cluster 5.2 - 5.4 whatever its size; at 2047 rows 16-block
// clusters 6.2, 37 blocks and a merge 7.4; at 8191 rows 10.0 and 9.7.  Clusters in front of a merge only add
// their cost (11 - 13 us there).
#pragma once

#include <cstring>
#include <mutex>

#include "decode_shared.cuh"

namespace tc {

// The new token's K/V row (and, in the dense models, the rotation of K and of q in place), done by the decode
// launch itself.  All pointers are nullable.
struct NewToken {
    const float *k, *v;       // f32 [nKV][hd]: stored into row len - 1 before it is attended
    const float *cosT, *sinT; // [rows][hd / 2]: K of the new row and q are rotated by table row len - 1
    float *qRot;              // where the rotated q goes (q itself: the rotation is in place)
    float *mirrorK, *mirrorV; // int8 stores with an f32 store beside them: its rows (written verbatim)
    uint64_t mirrorRows;
};

// What a decode (or causal-rows) launch over an f32 / fp16 store is told.
struct DecodeKvParams {
    const float *q;
    float *out;
    float *pAcc, *pM, *pL;
    const uint32_t *devPos;  // nullable: position read at kernel time
    void *kvK, *kvV;         // the store
    uint64_t totalRows;
    uint32_t lenHost;        // rows to attend; with devPos their upper bound
    uint32_t nHeads, nKV, group;
    uint32_t colBase;        // decode: the 8 MMA columns are q heads colBase .. colBase + 7 of the kv head
    uint32_t chunkTokens, numChunks;
    uint32_t qRows, cachePos;  // causal rows: row s sees cache rows [0, cachePos + s], 8 rows of a q head per block
    float invSqrt;
    int directOut, kvHalf;
    NewToken tok;            // decode: the row this launch appends first
    unsigned int *err;
};

// ---- the split ------------------------------------------------------------------------------
struct ClusterPlan {
    uint32_t cluster;      // blocks per cluster
    uint32_t clusters;     // clusters per kv head = partial slots used (1: direct output); more than one: of one block each
    uint32_t chunkTokens;  // tokens per block, a multiple of 16
};

// What the plan weighs.  maxClusters[i]: clusters of 2^i blocks that are resident at once
// (cudaOccupancyMaxActiveClusters: 16-block clusters lose the SMs of a GPC that do not make up a whole one).
struct ClusterCost {
    float tileUs;       // a warp's time for one 16-token tile
    float smTileUs;     // an SM's, with its warps busy
    uint32_t warps;     // warps of a block: tile j goes to warp j % warps
    uint32_t tileBytes; // K and V bytes of a tile
    uint32_t maxClusters[5];
};

// The fewest-microseconds split among one cluster of 1 - 16 blocks per kv head and n blocks with a merge behind them:
// the tiles a warp has to do one after the other, the tiles of an SM or the HBM stream, whichever takes longest, plus
// what the fold costs (0.5 us in a cluster, 2.5 us as a merge launch and a little more from the 33rd partial on), and 3 us for what a
// block does ahead of its first tile and behind its last one where clusters take turns.  (With 1.7 us for the merge and nothing for
// turns, per layer -> like this: fp16, 28 / 4 / 128 at 12000 rows 10.5 -> 8.9 us, 12 / 2 / 128 at 4500 6.7 -> 6.0, 40 / 8 / 128 at 5500 / 9000 10.3 /
// 12.6 -> 8.4 / 11.0, 14 / 2 / 64 at 7000 6.7 -> 5.7; f32, 14 / 2 / 64 at 2500 7.6 -> 6.4.  With 3.4 us for the merge: 28 / 4 / 128 at 20000
// 12.9 -> 11.9, 8 / 2 / 128 at 11000 7.6 -> 8.4.)
inline ClusterPlan searchClusterPlan(uint32_t nKV, uint32_t maxLen, uint32_t slots, bool needPartials, const ClusterCost &c) {
    const uint32_t tiles = maxLen == 0 ? 1u : (maxLen + 15) / 16, sms = static_cast<uint32_t>(numSMs());
    const float stream = static_cast<float>(tiles) * static_cast<float>(nKV) * static_cast<float>(c.tileBytes) * (1.0f / 5.6e6f);
    auto workUs = [&](uint32_t perBlock, uint32_t blocks, uint32_t waves) {
        const float warp = static_cast<float>((perBlock + c.warps - 1) / c.warps * waves) * c.tileUs;
        const float sm = static_cast<float>(perBlock * ((blocks + sms - 1) / sms)) * c.smTileUs;
        return warp > sm ? (warp > stream ? warp : stream) : (sm > stream ? sm : stream);
    };
    ClusterPlan best = {1, 1, tiles * 16};
    float bestUs = 1e30f;
    auto consider = [&](uint32_t size, uint32_t n, float us) {
        if (us >= bestUs) return;
        bestUs = us;
        best.cluster = size;
        best.clusters = n;
        best.chunkTokens = (tiles + n * size - 1) / (n * size) * 16;
    };
    const float merge = needPartials ? 2.5f : 0.0f;
    for (uint32_t lg = 0; lg < 5; ++lg) {
        const uint32_t size = 1u << lg;
        if (c.maxClusters[lg] == 0 || (lg > 0 && size / 2 >= tiles)) continue;
        const uint32_t turns = (nKV + c.maxClusters[lg] - 1) / c.maxClusters[lg];
        consider(size, 1, workUs((tiles + size - 1) / size, size * nKV, turns) + 3.0f * (turns - 1u) + (lg > 0 ? 0.45f + 0.03f * lg : 0.0f) + merge);
    }
    uint32_t most = c.maxClusters[0] / nKV;  // blocks per kv head in one wave
    most = most > slots ? slots : most;
    for (uint32_t n = 2; n <= most && n <= tiles; ++n) {
        const uint32_t perBlock = (tiles + n - 1) / n;
        if ((tiles + perBlock - 1) / perBlock != n) continue;  // the last blocks would have no rows
        consider(1, n, workUs(perBlock, n * nKV, 1) + 2.5f + (n > 32 ? 0.035f * (n - 32) : 0.0f));
    }
    return best;
}

// The search takes about a microsecond of the host, a token's layers ask the same question one after the other: each
// thread keeps its last answer per kernel (`slot`).
inline ClusterPlan planCluster(uint32_t slot, uint32_t nKV, uint32_t maxLen, uint32_t slots, bool needPartials,
                               const ClusterCost &c) {
    struct Last {
        uint32_t nKV, tiles, slots, needPartials;
        ClusterCost cost;
        ClusterPlan plan;
    };
    static thread_local Last last[8];
    Last &l = last[slot & 7u];
    const uint32_t tiles = (maxLen + 15) / 16;
    if (l.nKV != nKV || l.tiles != tiles || l.slots != slots || l.needPartials != (needPartials ? 1u : 0u) ||
        memcmp(&l.cost, &c, sizeof(c)) != 0) {
        l.plan = searchClusterPlan(nKV, maxLen, slots, needPartials, c);
        l.nKV = nKV, l.tiles = tiles, l.slots = slots, l.needPartials = needPartials ? 1u : 0u, l.cost = c;
    }
    return l.plan;
}

// f32 (decode_kv.cu) and fp16 (decode_kv16.cu) stores, one query row: arguments of tc_attn_decode_kv plus the new token
int decodeKvToken(const float *q, const void *kvK, const void *kvV, float *attnOut, float *pAcc, float *pM, float *pL,
                  uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t pos, const uint32_t *devPos, uint64_t totalRows,
                  uint32_t numChunks, float invSqrt, int kvHalf, uint8_t *q81Out, const NewToken &tok, cudaStream_t st);
int decodeKv16(const DecodeKvParams &prm, uint32_t hd, uint8_t *q81Out, cudaStream_t st);
int prefillKv16(DecodeKvParams prm, uint32_t hd, cudaStream_t st);
// causal rows over either store in blocks of 32 (prefill_exact.cu), and whether they beat the 8-row form; arguments
// already validated
bool prefillExactWins(uint32_t rows, uint64_t before, uint32_t nHeads, uint32_t hd, int kvHalf);
int prefillExact(const float *q, const void *kvK, const void *kvV, float *out, uint32_t seqLen, uint32_t nHeads,
                 uint32_t nKV, uint32_t hd, uint32_t cachePos, const uint32_t *devPos, uint64_t totalRows, float invSqrt,
                 int kvHalf, cudaStream_t st);

#ifdef __CUDACC__

// ---- a warp's tiles ------------------------------------------------------------------------------------
// 16 bytes global -> shared past L1; a warp's copies complete in the order of its commits.
__device__ __forceinline__ void cpAsync16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpAsyncWait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
    __syncwarp();
}
// ROWS rows of ROWB bytes (a multiple of 128) by one warp, from row `row` of a [rows][stride bytes] matrix on -- the first
// `count` of them: what lies behind is left as it is, and masked by the caller -- as ROWB / 128 boxes of [ROWS][128
// bytes], 16-byte units xor-swizzled by the row: what ldmatrix and 16-byte loads down the rows read without bank conflicts.
template <int ROWS, int ROWB>
__device__ __forceinline__ void copyTile(uint32_t dst, const uint8_t *base, uint32_t stride, uint64_t row, uint32_t count,
                                         uint32_t lane) {
    constexpr uint32_t U = ROWB / 16;  // 16-byte units per row
    if constexpr (U <= 32) {
        // a copy instruction of the warp covers R whole rows; from one to the next only constants are added
        constexpr uint32_t R = 32 / U;
        const uint32_t r0 = lane / U, u = lane % U;
        const uint32_t d0 = dst + (u / 8) * (ROWS * 128) + r0 * 128 + (((u & 7u) ^ (r0 & 7u)) << 4);
        const uint8_t *src = base + (row + r0) * stride + u * 16;
        if (count >= ROWS) {
#pragma unroll
            for (uint32_t k = 0; k < ROWS / R; ++k) {
                cpAsync16((d0 ^ (((k * R) & 7u) << 4)) + k * R * 128, src);
                src += R * stride;
            }
        } else {
#pragma unroll
            for (uint32_t k = 0; k < ROWS / R; ++k) {
                if (r0 + k * R < count) cpAsync16((d0 ^ (((k * R) & 7u) << 4)) + k * R * 128, src);
                src += R * stride;
            }
        }
    } else {
        constexpr uint32_t N = U / 32;  // copy instructions per row
        const uint8_t *src = base + row * stride + lane * 16;
#pragma unroll
        for (uint32_t r = 0; r < ROWS; ++r) {
#pragma unroll
            for (uint32_t k = 0; k < N; ++k) {
                const uint32_t u = k * 32 + lane;
                if (r < count) cpAsync16(dst + (u / 8) * (ROWS * 128) + r * 128 + (((u & 7u) ^ (r & 7u)) << 4), src + k * 512);
            }
            src += stride;
        }
    }
}
// Where byte `off` of row r of such a tile lies.
template <int ROWS>
__device__ __forceinline__ uint32_t tileOffset(uint32_t r, uint32_t off) {
    return (off >> 7) * (ROWS * 128) + r * 128 + ((((off >> 4) & 7u) ^ (r & 7u)) << 4) + (off & 15u);
}

// The rows of one 16-token tile of K and V (ROWB bytes each) towards L2, by one warp.  Right at any time, also ahead of the
// dependency wait: a row that a kernel in flight still writes is read after the wait.  The launches of a token's
// layers overlap by their prologues, so DRAM streams the next layer's rows while this one computes.
template <int ROWB>
__device__ __forceinline__ void prefetchTile(const uint8_t *k, const uint8_t *v, size_t stride, uint64_t row, uint64_t lastRow,
                                             uint32_t lane) {
    const uint64_t r = row + (lane & 15u);
    const uint8_t *p = (lane < 16u ? k : v) + (r < lastRow ? r : lastRow) * stride;
#pragma unroll
    for (int i = 0; i < ROWB / 128; ++i) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i * 128));
}
constexpr uint32_t kPrefetchTiles = 2;  // of a warp, ahead of the wait

// What a token brings along (prefetchL2 in tc_common.cuh), a line per thread: `heads` vectors of q, the rows of a kv head to append
// and -- with a host length -- the table row that rotates them.  Cold, they came out of DRAM behind the wait.
template <int HD>
__device__ __forceinline__ void prefetchToken(const float *q, uint32_t heads, const float *k, const float *v, const float *cosRow,
                                              const float *sinRow, uint32_t thread) {
    constexpr uint32_t L = HD / 32;  // lines of a row
    const uint32_t i = thread - heads * L;
    if (thread < heads * L) prefetchL2(q + 32u * thread);
    else if (i < 2u * L && k != nullptr) prefetchL2((i < L ? k : v) + 32u * (i % L));
    else if (i >= 2u * L && i < 3u * L && cosRow != nullptr) prefetchL2((i % L < L / 2u ? cosRow : sinRow) + 32u * (i % (L / 2u)));
}

// ---- distributed shared memory -------------------------------------------------------------------
__device__ __forceinline__ uint32_t clusterRank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t clusterSize() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void clusterSync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// "This block runs": the other blocks may write its shared memory once they have waited for it.
__device__ __forceinline__ void clusterHello() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void clusterHelloWait() { asm volatile("barrier.cluster.wait;" ::: "memory"); }
__device__ __forceinline__ uint32_t mapRank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// The rotated q of nValid heads, written in place: pairs [first, ...) of the heads, a share per caller.
// x0' = fmaf(x0, c, -(x1 s)), x1' = fmaf(x0, s, x1 c): the arithmetic of kvAppendKernel, bit for bit.
template <int HD>
__device__ __forceinline__ void rotateQ(float *q, const float *cosT, const float *sinT, uint32_t tableRow, uint32_t nValid,
                                        uint32_t first, uint32_t step) {
    constexpr uint32_t H = HD / 2;
    for (uint32_t i = first; i < nValid * H; i += step) {
        float *x = q + static_cast<size_t>(i / H) * HD + i % H;
        const float c = __ldg(cosT + static_cast<size_t>(tableRow) * H + i % H);
        const float s = __ldg(sinT + static_cast<size_t>(tableRow) * H + i % H);
        const float x0 = x[0], x1 = x[H];
        x[0] = fmaf(x0, c, -__fmul_rn(x1, s));
        x[H] = fmaf(x0, s, __fmul_rn(x1, c));
    }
}

// ---- the fold -----------------------------------------------------------------------------------------
struct FoldTarget {
    float *out, *pAcc, *pM, *pL;
    uint32_t numChunks, slot;   // slot stride of the partials, this cluster's slot
    uint32_t firstHead, nValid; // q heads (index of the first one's vector) this block's columns stand for
    int direct;                 // normalise and write `out`; else write the partial
    float *qRot;                // nullable: q of the first head, to be rotated in place once every block has read it
    const float *cosT, *sinT;
    uint32_t tableRow;
};

template <int HD>
__device__ __forceinline__ void foldStore(const FoldTarget &f, uint32_t j, uint32_t d4, float M, float l, float4 acc) {
    const size_t o = static_cast<size_t>(f.firstHead) + j;
    if (f.direct) {
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        *reinterpret_cast<float4 *>(f.out + o * HD + 4 * d4) = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    } else {
        const size_t p = o * f.numChunks + f.slot;
        *reinterpret_cast<float4 *>(f.pAcc + p * HD + 4 * d4) = acc;
        if (d4 == 0) {
            // natural-log units: the merge contract is w = exp2((m - M) * log2e)
            f.pM[p] = M > -1e29f ? M * 0.6931471805599453f : kNegBig;
            f.pL[p] = l;
        }
    }
}

// The blocks of a cluster share the output: rank r takes the r-th slice of its nValid x HD / 4 float4s (`per` of them), and
// every block writes its results for that slice into rank r's inbox.  One cluster barrier lies between the writes and the
// reads (which are local); a block may leave after it.  (With the results read from the other blocks' memory instead it
// took a round trip and a second barrier more: 0.5 us of a launch.)
template <int V4>
struct FoldInbox {
    float4 acc[8 * V4 + 16];
    float2 ml[8 * V4 + 16];
};
template <int V4>
__device__ __forceinline__ void inboxPush(FoldInbox<V4> &in, uint32_t idx, uint32_t per, uint32_t rank, float M, float l,
                                          float4 acc) {
    const uint32_t owner = idx / per, at = rank * per + (idx - owner * per);
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(mapRank(smemAddr(&in.acc[at]), owner)), "f"(acc.x),
                 "f"(acc.y), "f"(acc.z), "f"(acc.w)
                 : "memory");
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(mapRank(smemAddr(&in.ml[at]), owner)), "f"(M), "f"(l) : "memory");
}
template <int V4>
__device__ __forceinline__ void inboxTake(const FoldInbox<V4> &in, uint32_t i, uint32_t per, uint32_t n, float &M, float &l,
                                          float4 &acc) {
    M = kNegBig, l = 0.0f, acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t r = 0; r < n; ++r) M = fmaxf(M, in.ml[r * per + i].x);
#pragma unroll 4
    for (uint32_t r = 0; r < n; ++r) {
        const float2 ml = in.ml[r * per + i];
        const float4 a = in.acc[r * per + i];
        const float wgt = fastExp2(ml.x - M);
        l = fmaf(wgt, ml.y, l);
        acc.x = fmaf(wgt, a.x, acc.x);
        acc.y = fmaf(wgt, a.y, acc.y);
        acc.z = fmaf(wgt, a.z, acc.z);
        acc.w = fmaf(wgt, a.w, acc.w);
    }
}

// A warp's results in shared memory: [8 columns][kRow] accumulators, m[8] (log2 units), l[8].  The row stride keeps the four
// columns that a warp stores at a time in different banks (rows of HD floats put them into the same ones: a four-way
// conflict: 0.15 - 0.6 us of a decode call, the most at head_dim 256).
template <int HD>
struct FoldScratch {
    static constexpr int kRow = HD + 4, kM = 8 * kRow, kL = kM + 8, kWarp = kL + 8;
};

// Every warp has left its results in its part of scr ([NW][FoldScratch::kWarp]).  Called by all THREADS threads of the block
// (tid) with the warps' parts complete; in a cluster every thread has said clusterHello() before.
template <int HD, int NW, int THREADS = NW * 32>
__device__ __forceinline__ void clusterFold(const float *scr, const FoldTarget &f, uint32_t tid) {
    using F = FoldScratch<HD>;
    constexpr uint32_t kWarpScr = F::kWarp, V4 = HD / 4;
    __shared__ FoldInbox<V4> inbox;
    const uint32_t n = clusterSize(), rank = clusterRank();
    const uint32_t total = f.nValid * V4, per = (total + n - 1) / n;
    if (n > 1) clusterHelloWait();
    for (uint32_t idx = tid; idx < total; idx += THREADS) {
        const uint32_t d4 = idx % V4, j = idx / V4;
        float M = kNegBig;
#pragma unroll
        for (int w = 0; w < NW; ++w) M = fmaxf(M, scr[w * kWarpScr + F::kM + j]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float l = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const float *s = scr + w * kWarpScr;
            const float wgt = fastExp2(s[F::kM + j] - M);
            l = fmaf(wgt, s[F::kL + j], l);
            const float4 a = *reinterpret_cast<const float4 *>(s + j * F::kRow + 4 * d4);
            acc.x = fmaf(wgt, a.x, acc.x);
            acc.y = fmaf(wgt, a.y, acc.y);
            acc.z = fmaf(wgt, a.z, acc.z);
            acc.w = fmaf(wgt, a.w, acc.w);
        }
        if (n == 1) foldStore<HD>(f, j, d4, M, l, acc);
        else inboxPush<V4>(inbox, idx, per, rank, M, l, acc);
    }
    if (n > 1) clusterSync();
    // (in a cluster of one block the caller's barrier has every warp's q in registers)
    if (f.qRot != nullptr)
        rotateQ<HD>(f.qRot, f.cosT, f.sinT, f.tableRow, f.nValid, rank * THREADS + tid, n * THREADS);
    if (n == 1) return;
    for (uint32_t i = tid; i < per && rank * per + i < total; i += THREADS) {
        const uint32_t idx = rank * per + i;
        float M, l;
        float4 acc;
        inboxTake<V4>(inbox, i, per, n, M, l, acc);
        foldStore<HD>(f, idx / V4, idx % V4, M, l, acc);
    }
}

// ---- the new token's row ---------------------------------------------------------------------------------
template <typename KVT>
__device__ __forceinline__ KVT kvElem(float x) {
    if constexpr (sizeof(KVT) == 2) return __float2half_rn(x);
    else return x;
}

// The new token's K and V row of one kv head, by one warp: loaded ahead of the query's preparation, stored behind it -- into
// the store and, when the warp's tile with that row is among the first ones (`tileK` / `tileV`, row r of them), into that
// tile: the row does not go through memory on its way there.  A later tile's copies read it back.
//
// f32 / fp16 stores: V verbatim, K rotated NEOX-style when there are tables (x0' = fmaf(x0, c, -(x1 s)), x1' = fmaf(x0, s, x1
// c)): the arithmetic of kvAppendKernel, bit for bit.
template <int HD>
struct NewRow {
    static constexpr int N = HD / 64;
    float k0[N], k1[N], v0[N], v1[N], c[N], s[N];
    __device__ __forceinline__ void load(const NewToken &t, uint32_t kvHead, uint32_t tableRow, uint32_t lane) {
        const float *k = t.k + static_cast<size_t>(kvHead) * HD, *v = t.v + static_cast<size_t>(kvHead) * HD;
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const uint32_t j = lane + 32 * i;
            k0[i] = k[j], k1[i] = k[j + HD / 2], v0[i] = v[j], v1[i] = v[j + HD / 2];
            if (t.cosT != nullptr) {
                c[i] = __ldg(t.cosT + static_cast<size_t>(tableRow) * (HD / 2) + j);
                s[i] = __ldg(t.sinT + static_cast<size_t>(tableRow) * (HD / 2) + j);
            }
        }
    }
    template <typename KVT>
    __device__ __forceinline__ void store(bool rotate, KVT *kRow, KVT *vRow, uint8_t *tileK, uint8_t *tileV, uint32_t r,
                                          uint32_t lane) const {
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            const uint32_t j = lane + 32 * i, j2 = j + HD / 2;
            float a = k0[i], b = k1[i];
            if (rotate) {
                a = fmaf(k0[i], c[i], -__fmul_rn(k1[i], s[i]));
                b = fmaf(k0[i], s[i], __fmul_rn(k1[i], c[i]));
            }
            const KVT ka = kvElem<KVT>(a), kb = kvElem<KVT>(b), va = kvElem<KVT>(v0[i]), vb = kvElem<KVT>(v1[i]);
            kRow[j] = ka, kRow[j2] = kb;
            vRow[j] = va, vRow[j2] = vb;
            if (tileK != nullptr) {
                const uint32_t o = tileOffset<16>(r, j * sizeof(KVT)), o2 = tileOffset<16>(r, j2 * sizeof(KVT));
                *reinterpret_cast<KVT *>(tileK + o) = ka, *reinterpret_cast<KVT *>(tileK + o2) = kb;
                *reinterpret_cast<KVT *>(tileV + o) = va, *reinterpret_cast<KVT *>(tileV + o2) = vb;
            }
        }
    }
};

// int8 pools: quantised (the arithmetic of kvQuantKernel), with its scale; mirK / mirV (nullable): an f32 store's rows that
// get it verbatim.
template <int HD, int T>
struct NewQuantRow {
    static constexpr int N = HD / 128;
    float4 kx[N], vx[N];
    __device__ __forceinline__ void load(const float *k, const float *v, uint32_t lane) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            kx[i] = __ldg(reinterpret_cast<const float4 *>(k) + lane + 32 * i);
            vx[i] = __ldg(reinterpret_cast<const float4 *>(v) + lane + 32 * i);
        }
    }
    __device__ __forceinline__ void store(uint32_t *kRow, uint32_t *vRow, float *ksp, float *vsp, float4 *mirK, float4 *mirV,
                                          uint8_t *tileK, uint8_t *tileV, float *scaleK, float *scaleV, uint32_t r,
                                          uint32_t lane) const {
        float mk = 0.0f, mv = 0.0f;
        auto amax4 = [](const float4 &x) { return fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))); };
#pragma unroll
        for (int i = 0; i < N; ++i) {
            mk = fmaxf(mk, amax4(kx[i]));
            mv = fmaxf(mv, amax4(vx[i]));
            if (mirK != nullptr) mirK[lane + 32 * i] = kx[i], mirV[lane + 32 * i] = vx[i];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            mk = fmaxf(mk, __shfl_xor_sync(0xffffffffu, mk, o));
            mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
        }
        const float sk = mk > 0.0f ? __fdiv_rn(mk, 127.0f) : 1.0f, sv = mv > 0.0f ? __fdiv_rn(mv, 127.0f) : 1.0f;
        if (lane == 0) {
            *ksp = sk, *vsp = sv;
            if (tileK != nullptr) scaleK[r] = sk, scaleV[r] = sv;
        }
        auto q8 = [](float x, float sc) -> uint32_t {
            int qv = __float2int_rn(__fdiv_rn(x, sc));
            qv = qv < -128 ? -128 : (qv > 127 ? 127 : qv);
            return static_cast<uint32_t>(qv) & 0xffu;
        };
        auto pack = [&](const float4 &x, float sc) {
            return q8(x.x, sc) | (q8(x.y, sc) << 8) | (q8(x.z, sc) << 16) | (q8(x.w, sc) << 24);
        };
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t w = pack(kx[i], sk), w2 = pack(vx[i], sv), o = tileOffset<T>(r, 4 * (lane + 32 * i));
            kRow[lane + 32 * i] = w;
            vRow[lane + 32 * i] = w2;
            if (tileK != nullptr) *reinterpret_cast<uint32_t *>(tileK + o) = w, *reinterpret_cast<uint32_t *>(tileV + o) = w2;
        }
    }
};

// A kernel's shared-memory and cluster attributes, set once per device, and how many clusters of each size are
// resident at once (the answer depends on its shared memory).
struct ClusterSetup {
    std::mutex mu;
    bool done[64] = {false};
    uint32_t maxClusters[64][5];
};
template <typename K>
int setupCluster(ClusterSetup &s, K kern, uint32_t threads, size_t smem, const uint32_t **limits) {
    int dev = 0;
    TC_CUDA_OK(cudaGetDevice(&dev));
    TC_REQUIRE(dev >= 0 && dev < 64, TC_EUNSUPPORTED, "device ordinal %d", dev);
    std::lock_guard<std::mutex> lk(s.mu);
    if (!s.done[dev]) {
        TC_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        TC_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        for (uint32_t lg = 0; lg < 5; ++lg) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1u << lg);
            cfg.blockDim = dim3(threads);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 1u << lg;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            TC_CUDA_OK(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
            s.maxClusters[dev][lg] = static_cast<uint32_t>(n);
        }
        s.done[dev] = true;
    }
    *limits = s.maxClusters[dev];
    return TC_OK;
}

// Plan and launch of the f32 / fp16 decode kernels.
template <typename K>
int launchKvDecode(ClusterSetup &setup, K kern, uint32_t threads, size_t smem, uint32_t hd, uint32_t warps,
                   uint32_t tileBytes, float tileUs, float smTileUs, DecodeKvParams prm, uint8_t *q81Out, cudaStream_t st) {
    const uint32_t *limits = nullptr;
    int rc = setupCluster(setup, kern, threads, smem, &limits);
    if (rc != TC_OK) return rc;
    ClusterCost cost = {tileUs, smTileUs, warps, tileBytes, {}};
    memcpy(cost.maxClusters, limits, sizeof(cost.maxClusters));
    // (a caller without partial buffers has one cluster per kv head, wherever the line to the merge lies)
    const bool partials = prm.pAcc && prm.pM && prm.pL;
    const ClusterPlan pl = planCluster(hd / 64u + (prm.kvHalf ? 4u : 0u), prm.nKV, prm.lenHost, partials ? prm.numChunks : 1u,
                                       q81Out != nullptr, cost);
    prm.directOut = pl.clusters == 1 && q81Out == nullptr ? 1 : 0;
    prm.chunkTokens = pl.chunkTokens;
    if (!prm.directOut)
        TC_REQUIRE(partials, TC_EWORKSPACE, "tc_attn_decode_kv: partial buffers are required");
    // several clusters read q: the merge writes its rotation behind them
    QRotation rot = {nullptr, nullptr, nullptr, prm.lenHost};
    if (prm.tok.qRot != nullptr && !prm.directOut) {
        rot.q = prm.tok.qRot, rot.cosT = prm.tok.cosT, rot.sinT = prm.tok.sinT;
        prm.tok.qRot = nullptr;
    }
    for (uint32_t cb = 0; cb < prm.group; cb += 8) {  // 8 q heads of a kv head per launch
        prm.colBase = cb;
        if (cb) prm.tok.k = prm.tok.v = nullptr;      // the row is in
        rc = launchDependent(kern, dim3(pl.clusters * pl.cluster, prm.nKV, 1), threads, smem, st, pl.cluster, prm);
        if (rc != TC_OK) return rc;
    }
    if (prm.directOut) return TC_OK;
    return launchMerge(prm.pAcc, prm.pM, prm.pL, prm.out, 1, prm.nHeads, prm.numChunks, pl.clusters, hd, prm.devPos,
                       prm.devPos ? 1u : 0u, 0u, q81Out, true, st, 0, 0, rot);
}

#endif  // __CUDACC__

}  // namespace tc
