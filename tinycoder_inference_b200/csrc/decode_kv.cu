// decode_kv.cu -- grouped-query attention over an f32 KV cache: split-KV decode
// and, with query rows as columns, the unsplit causal kernel.
//
// What it replaces: launchDecodeAttentionSplit / kWarpAttentionSplit +
// kAttnCombinePartial(W4) and kWarpAttention / kWarpAttentionPos of the reference
// (include/gpu/GpuAttentionKernels.hpp:211-272, 537-599, 625-766, 909-1230), and
// (the fp16 cache, kvHalf, is served by the twin kernel in decode_kv16.cu) and
// the f32 twins kQ35WarpAttention / kQ35StoreKV-fed split path of the hybrid
// models (include/gpu/GpuQwen35Kernels.hpp:2437-2492): score = dot(q, k) *
// invSqrt, online softmax with exp2, out = sum p v / sum p, all f32.
//
// A block streams a token range of one kv head; its warps take 16-token tiles in
// turn, each with copies and slots of its own, and serve every q head of the kv head.  The split
// over clusters of blocks, the fold of their results and the new token's row are
// decode_cluster.cuh's.  The arithmetic differs from the int8 kernel's: K and V are
// arbitrary f32, so QK^T and PV run as 3xTF32 tensor-core products
// (mma.sync.m16n8k8: x = hi + lo with both parts tf32; hi*hi + lo*hi + hi*lo keeps
// ~21 mantissa bits and the full f32 exponent range, f32 accumulation).  f32 rows
// are four times the bytes of int8 rows, so per byte this costs a quarter of the
// instructions and the kernel stays HBM-bound.
#include "decode_cluster.cuh"

namespace tc {

// Every warp has SLOTS slots for 16-token tiles of K and as many of V, each as HD / 32 boxes of [16 rows][32 floats].
template <int HD, int NW, int SLOTS, bool SHAREQ>
struct DecodeKvSmem {
    static constexpr int NB = HD / 32;             // 32-float boxes per row
    static constexpr int kTileBytes = 16 * HD * 4; // K (or V) bytes of a tile
    static constexpr int kSlots = NW * SLOTS * 2 * kTileBytes, kScratch = NW * FoldScratch<HD>::kWarp * 4;  // (the fold reuses the slots)
    static constexpr int kQuery = kSlots > kScratch ? kSlots : kScratch;   // decode: the block's query operands
    static constexpr int kTotal = kQuery + (SHAREQ ? HD * 64 : 0) + 128;
    static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

constexpr bool kvSharesQuery(int hd, int blocksPerSm, bool rows) { return !rows && hd >= 128 && blocksPerSm == 1; }

__device__ __forceinline__ void splitTf32(float x, uint32_t &hi, uint32_t &lo) {
    hi = toTf32(x);
    lo = toTf32(x - __uint_as_float(hi));
}

// ROWS: the causal kernel (one block per 8 query rows and q head); otherwise decode, blocks of a cluster
// share a kv head's tokens.
//
// What bounds it: a warp needs about 800 instructions and six dependent chains of tensor-core products for 16
// tokens (1 - 2 us alone), HBM delivers 16 tokens of one kv head to an SM in 0.4 us at head_dim 128: it takes
// many warps per SM, each with a tile of its own, to keep up.  16-byte copies by the warp itself serve that: small TMA
// boxes from one producer thread do not (22 us for 18.8 MB of one layer), and boxes shared by a block's warps leave
// too few of them (17 us; this form 15).  192 MB of one layer (28 / 4 / 128 at 47000 rows): 42 us.
template <int HD, int NW, int SLOTS, int BPS, bool ROWS>
__global__ void __launch_bounds__(NW * 32, BPS) decodeKvKernel(const __grid_constant__ DecodeKvParams p) {
    // The block's warps prepare the query together, but where it is cheap (head_dim 64) or registers and shared memory are short
    // (two blocks per SM).  One of head_dim 256 stays in shared memory: 128 registers, and the spills that came with them.
    // 28 / 4 / 128, per layer: 2047 rows 7.85 -> 7.65 us, 8191 rows 14.85 -> 14.6; 16 / 4 / 256 (norm and gate included) 14000
    // rows 40.9 -> 35.8, 20000 rows 54.6 -> 45.0.
    constexpr bool kShareQuery = kvSharesQuery(HD, BPS, ROWS), kQueryInRegs = HD <= 128 || !kShareQuery;
    using L = DecodeKvSmem<HD, NW, SLOTS, kShareQuery>;
    constexpr int T = 16, NB = L::NB;
    constexpr int KS = HD / 8;   // tf32 k-steps of the QK product
    constexpr int MTO = HD / 16;  // 16-dim output tiles

    const uint32_t chunk = blockIdx.x, hg = blockIdx.y, b = ROWS ? gridDim.z - 1u - blockIdx.z : blockIdx.z;  // (late rows first)
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;

    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 127) & ~uintptr_t(127));
    constexpr bool kOwnScratch = !kShareQuery || !kQueryInRegs;  // else where the query operands were
    __shared__ float pScratch[kOwnScratch ? NW : 1][16 * 8];

    if (!ROWS) {
        // (a device position read here may be a step old: good enough to know which rows to pull)
        const uint32_t hint = p.devPos ? min(p.devPos[0], p.lenHost - 1u) + 1u : p.lenHost;
        const uint32_t per = p.devPos ? tokensPerBlock(hint, gridDim.x) : p.chunkTokens;
        const uint8_t *k = static_cast<const uint8_t *>(p.kvK) + static_cast<size_t>(hg) * HD * 4;
        const uint8_t *v = static_cast<const uint8_t *>(p.kvV) + static_cast<size_t>(hg) * HD * 4;
        for (uint32_t i = 0, tok = chunk * per + warp * T; i < kPrefetchTiles && tok < min(hint, (chunk + 1u) * per); ++i, tok += NW * T)
            prefetchTile<HD * 4>(k, v, static_cast<size_t>(p.nKV) * HD * 4, tok, p.totalRows - 1, lane);
        const size_t row = static_cast<size_t>(hg) * HD, table = static_cast<size_t>(p.lenHost - 1u) * (HD / 2);
        const bool rotates = p.tok.cosT != nullptr && p.devPos == nullptr;
        // (at head_dim 64, 15 - 20000 rows in a graph, with it / without: one layer 0.97 - 1.06 of the time, mean 1.00, four 0.98 - 1.01, eight 0.98 - 1.01,
        // mean 0.995, and 0.94 - 0.98 where the inputs are cold at half of the lengths)
        prefetchToken<HD>(p.q + (static_cast<size_t>(hg) * p.group + p.colBase) * HD, min(8u, p.group - p.colBase),
                          p.tok.k != nullptr ? p.tok.k + row : nullptr, p.tok.v + row, rotates ? p.tok.cosT + table : nullptr,
                          p.tok.sinT + table, threadIdx.x);
    }
    gridDepWait();
    gridDepLaunch();

    uint32_t pos = p.devPos ? p.devPos[0] : 0u;
    uint32_t len, rowsPos = p.cachePos;
    if (ROWS) {
        if (p.devPos) rowsPos = pos;
        len = rowsPos + min(p.qRows, b * 8u + 8u);
    } else {
        len = p.devPos ? min(pos, p.lenHost - 1u) + 1u : p.lenHost;  // (the host's length is the upper bound)
    }
    // A launch sized for a window shares the rows there are among all its blocks; the merge counts them the same way.
    const uint32_t share = ROWS ? len : (p.devPos ? tokensPerBlock(len, gridDim.x) : p.chunkTokens);
    const uint32_t t0 = ROWS ? 0u : chunk * share;
    if (!ROWS && t0 >= len && clusterSize() == 1) return;
    if (!ROWS && clusterSize() > 1) clusterHello();
    const uint32_t t1 = min(len, t0 + share);
    const uint32_t nTiles = t0 < t1 ? (t1 - t0 + T - 1) / T : 0u;
    const uint32_t kvHead = ROWS ? hg / p.group : hg;

    // Tile j belongs to warp j % NW, its slot (j / NW) % SLOTS.  A warp copies its own tiles: with one slot the
    // next tile's K while it works on this one's V and the next V while it works on K.
    auto slotK = [&](uint32_t i) { return smem + (warp * SLOTS + i % SLOTS) * 2 * L::kTileBytes; };
    const uint32_t stride = p.nKV * HD * 4;
    const uint8_t *storeK = static_cast<const uint8_t *>(p.kvK) + static_cast<size_t>(kvHead) * HD * 4;
    const uint8_t *storeV = static_cast<const uint8_t *>(p.kvV) + static_cast<size_t>(kvHead) * HD * 4;
    // the warp that takes the last tile stores the token's row; into the tile itself when that is among its first ones
    const bool append = !ROWS && p.tok.k != nullptr && t1 == len && nTiles != 0;
    const bool outside = append && p.devPos && pos >= p.totalRows;  // a device position outside the store: no row written
    if (outside && threadIdx.x == 0) atomicOr(p.err, kDevErrRowBound);
    const bool mine = append && !outside && (nTiles - 1u) % NW == warp;
    const bool intoTile = mine && (nTiles - 1u) / NW < SLOTS;
    const uint32_t have = intoTile ? len - 1u : static_cast<uint32_t>(min(static_cast<uint64_t>(len), p.totalRows));
    auto request = [&](uint32_t i, bool isV) {
        const uint32_t j = warp + i * NW, row = t0 + j * T;
        if (j < nTiles)
            copyTile<T, HD * 4>(smemAddr(slotK(i) + (isV ? L::kTileBytes : 0)), isV ? storeV : storeK, stride, row,
                                have > row ? have - row : 0u, lane);
        cpAsyncCommit();
    };
    auto requestK = [&](uint32_t i) { request(i, false); };
    auto requestV = [&](uint32_t i) { request(i, true); };
    NewRow<HD> fresh;
    // Behind the loads of q, which would queue behind the tiles' otherwise (28 / 4 / 128 at 2047 / 8191 rows 7.6 / 14.6 -> 7.45 / 13.8 us,
    // 16 / 4 / 256 at 2047 rows, norm and gate included, 16.9 -> 16.0) -- but at head_dim 64, where they are few (5.6 -> 5.7).
    auto requestFirst = [&]() {
        if (mine) fresh.load(p.tok, kvHead, len - 1u, lane);
#pragma unroll
        for (uint32_t i = 0; i < SLOTS; ++i) {
            requestK(i);
            requestV(i);
        }
    };

    const uint32_t g = lane >> 2, t = lane & 3u;
    auto colValid = [&](uint32_t j) { return ROWS ? (b * 8u + j < p.qRows) : (p.colBase + j < p.group); };
    auto colIndex = [&](uint32_t j) -> size_t {
        return ROWS ? (static_cast<size_t>(b) * 8u + j) * p.nHeads + hg
                    : static_cast<size_t>(kvHead) * p.group + p.colBase + j;
    };
    auto colLen = [&](uint32_t j) { return ROWS ? min(t1, rowsPos + b * 8u + j + 1u) : t1; };

    // q of column n = g as the B operand: k slot t / t+4 of step (bx, h, e) is
    // dim 32bx + 8t + 4h + 2e / +1 -- the order the swizzled 16-byte loads deliver.
    uint32_t qhi[kQueryInRegs ? KS : 1][2], qlo[kQueryInRegs ? KS : 1][2];
    const uint4 *frag = reinterpret_cast<const uint4 *>(smem + L::kQuery) + lane;  // [32-dim box][half][hi, lo][lane]
    if constexpr (!kShareQuery) {
        const bool valid = colValid(g);
        const float *qp = p.q + colIndex(valid ? g : 0) * HD;
        if constexpr (HD == 64) requestFirst();
        float4 qv[NB][2];
        // (plain loads: with a rotation q is written in place at the end of the launch)
#pragma unroll
        for (int bx = 0; bx < NB; ++bx)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                qv[bx][h] = valid ? *reinterpret_cast<const float4 *>(qp + 32 * bx + 8 * t + 4 * h)
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr (HD != 64) requestFirst();
        if (!ROWS && p.tok.cosT != nullptr) {
            // NEOX rotation: the partner of dim d is d + HD / 2, NB / 2 boxes further on
            const size_t row = static_cast<size_t>(len - 1u) * (HD / 2);
#pragma unroll
            for (int bx = 0; bx < NB / 2; ++bx)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int d = 32 * bx + 8 * t + 4 * h;
                    const float4 c = __ldg(reinterpret_cast<const float4 *>(p.tok.cosT + row + d));
                    const float4 s = __ldg(reinterpret_cast<const float4 *>(p.tok.sinT + row + d));
                    float4 &x = qv[bx][h], &y = qv[bx + NB / 2][h];
                    auto rot = [](float &x0, float &x1, float cc, float ss) {
                        const float a = fmaf(x0, cc, -__fmul_rn(x1, ss));
                        x1 = fmaf(x0, ss, __fmul_rn(x1, cc));
                        x0 = a;
                    };
                    rot(x.x, y.x, c.x, s.x);
                    rot(x.y, y.y, c.y, s.y);
                    rot(x.z, y.z, c.z, s.z);
                    rot(x.w, y.w, c.w, s.w);
                }
        }
#pragma unroll
        for (int bx = 0; bx < NB; ++bx)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 v = qv[bx][h];
                const int ks = (bx * 2 + h) * 2;
                splitTf32(v.x, qhi[ks][0], qlo[ks][0]);
                splitTf32(v.y, qhi[ks][1], qlo[ks][1]);
                splitTf32(v.z, qhi[ks + 1][0], qlo[ks + 1][0]);
                splitTf32(v.w, qhi[ks + 1][1], qlo[ks + 1][1]);
            }
    } else {
        // a column at a time each, four dims to a lane, the operands left where they are read
        uint4 *to = reinterpret_cast<uint4 *>(smem + L::kQuery);
        constexpr int QC = (8 + NW - 1) / NW, QI = (HD + 127) / 128;  // columns of a warp, float4s of a lane
        float4 qx[QC][QI], qy[QC][QI], qc[QI], qs[QI];
        const bool rotate = p.tok.cosT != nullptr;
#pragma unroll
        for (int k = 0; k < QC; ++k)
#pragma unroll
            for (int u = 0; u < QI; ++u) {
                const uint32_t j = warp + k * NW, i = lane + 32u * u;
                const bool upper = i >= HD / 8;
                const float *qp = p.q + colIndex(j < 8 && colValid(j) ? j : 0) * HD;
                // (plain loads: with a rotation q is written in place at the end of the launch)
                qx[k][u] = qy[k][u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j < 8 && colValid(j)) {
                    qx[k][u] = *reinterpret_cast<const float4 *>(qp + 4 * i);
                    if (rotate) qy[k][u] = *reinterpret_cast<const float4 *>(qp + 4 * (upper ? i - HD / 8 : i + HD / 8));
                }
                if (k == 0 && rotate) {
                    const size_t at = static_cast<size_t>(len - 1u) * (HD / 2) + 4 * (upper ? i - HD / 8 : i);
                    qc[u] = *reinterpret_cast<const float4 *>(p.tok.cosT + at), qs[u] = *reinterpret_cast<const float4 *>(p.tok.sinT + at);
                }
            }
        requestFirst();
#pragma unroll
        for (int k = 0; k < QC; ++k) {
            const uint32_t j = warp + k * NW;
            if (j >= 8) break;
#pragma unroll
            for (int u = 0; u < QI; ++u) {
                const uint32_t i = lane + 32u * u;
                float4 x = qx[k][u];
                if (rotate) {
                    // NEOX rotation: the partner of dim d is d + HD / 2
                    const bool upper = i >= HD / 8;
                    const float4 y = qy[k][u], c = qc[u], sn = qs[u];
                    auto rot = [upper](float own, float other, float cc, float ss) {
                        return upper ? fmaf(other, ss, __fmul_rn(own, cc)) : fmaf(own, cc, -__fmul_rn(other, ss));
                    };
                    x = make_float4(rot(x.x, y.x, c.x, sn.x), rot(x.y, y.y, c.y, sn.y), rot(x.z, y.z, c.z, sn.z),
                                    rot(x.w, y.w, c.w, sn.w));
                }
                uint4 hi, lo;
                splitTf32(x.x, hi.x, lo.x);
                splitTf32(x.y, hi.y, lo.y);
                splitTf32(x.z, hi.z, lo.z);
                splitTf32(x.w, hi.w, lo.w);
                // dims 4i ..: box i / 8, k slot (i % 8) / 2 of column j, half i % 2
                const uint32_t at = ((i / 8) * 4 + (i & 1u) * 2) * 32 + j * 4 + (i % 8) / 2;
                to[at] = hi, to[at + 32] = lo;
            }
        }
        __syncthreads();
        if constexpr (kQueryInRegs) {
#pragma unroll
            for (int k = 0; k < KS; k += 2) {
                const uint4 hi = frag[k * 32], lo = frag[(k + 1) * 32];
                qhi[k][0] = hi.x, qhi[k][1] = hi.y, qhi[k + 1][0] = hi.z, qhi[k + 1][1] = hi.w;
                qlo[k][0] = lo.x, qlo[k][1] = lo.y, qlo[k + 1][0] = lo.z, qlo[k + 1][1] = lo.w;
            }
            __syncthreads();  // (the warps' scratch for probabilities takes their place)
        }
    }
    const float cs = p.invSqrt * kLog2e;
    const uint32_t len0 = colLen(2 * t), len1 = colLen(2 * t + 1);

    if (mine) {
        const size_t at = (static_cast<size_t>(len - 1u) * p.nKV + kvHead) * HD;
        uint8_t *tile = intoTile ? slotK((nTiles - 1u) / NW) : nullptr;
        fresh.store(p.tok.cosT != nullptr, static_cast<float *>(p.kvK) + at, static_cast<float *>(p.kvV) + at, tile,
                    tile + L::kTileBytes, len - 1u - (t0 + (nTiles - 1u) * T), lane);
        __syncwarp();
    }

    // A tensor-core product drops the bits of its running sum that do not fit.  At head_dim 64, where one cluster for 2100 - 4100 rows leaves a
    // warp twice the tiles that a merge would, a tile's products are summed by themselves: 4000 rows are off by 4.1e-7 -> 3.3e-7 of the result's norm
    // (3.3e-7 with the merge), 30000 of 8 / 4 by 9.4e-7 -> 3.4e-7, in the same time (4000 rows 7.35 -> 7.32 us a layer in a graph, 30000 17.2 -> 17.3).
    constexpr bool kOwnSums = HD == 64 && !ROWS;
    float m0 = kNegBig, m1 = kNegBig, l0 = 0.0f, l1 = 0.0f;
    float o[MTO][4];
#pragma unroll
    for (int i = 0; i < MTO; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    static_assert(kOwnScratch || NW * 128 * 4 <= HD * 64, "scratch in place of the query operands");
    float *pS = kOwnScratch ? pScratch[kOwnScratch ? warp : 0] : reinterpret_cast<float *>(smem + L::kQuery) + warp * 128;

    for (uint32_t i = 0, tile = warp; tile < nTiles; ++i, tile += NW) {
        cpAsyncWait<2 * SLOTS - 1>();  // K of this tile is in, V may still be on its way
        const uint32_t tok0 = t0 + tile * T;
        const uint32_t tokA = tok0 + g, tokB = tokA + 8;

        // ---- S^T = K . Q^T (16 tokens x 8 columns), 3xTF32 ----
        // (two k steps in flight, the three products of a step in chains of their own)
        float sa[2][4] = {}, sb[2][4] = {}, sc[2][4] = {};
#pragma unroll
        for (int bx = 0; bx < NB; ++bx) {
            const uint8_t *kT = slotK(i) + bx * T * 128;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t off = ((2 * t + h) ^ g) << 4;
                const float4 xa = *reinterpret_cast<const float4 *>(kT + g * 128 + off);
                const float4 xb = *reinterpret_cast<const float4 *>(kT + (g + 8) * 128 + off);
                const int ks = (bx * 2 + h) * 2;
                uint4 qh, ql;
                if constexpr (kQueryInRegs) {
                    qh = make_uint4(qhi[ks][0], qhi[ks][1], qhi[ks + 1][0], qhi[ks + 1][1]);
                    ql = make_uint4(qlo[ks][0], qlo[ks][1], qlo[ks + 1][0], qlo[ks + 1][1]);
                } else {
                    qh = frag[ks * 32], ql = frag[(ks + 1) * 32];
                }
                {
                    uint32_t h0, l0_, h1, l1_, h2, l2_, h3, l3_;
                    splitTf32(xa.x, h0, l0_);
                    splitTf32(xb.x, h1, l1_);
                    splitTf32(xa.y, h2, l2_);
                    splitTf32(xb.y, h3, l3_);
                    mmaTf32(sa[0], h0, h1, h2, h3, qh.x, qh.y);
                    mmaTf32(sb[0], l0_, l1_, l2_, l3_, qh.x, qh.y);
                    mmaTf32(sc[0], h0, h1, h2, h3, ql.x, ql.y);
                }
                {
                    uint32_t h0, l0_, h1, l1_, h2, l2_, h3, l3_;
                    splitTf32(xa.z, h0, l0_);
                    splitTf32(xb.z, h1, l1_);
                    splitTf32(xa.w, h2, l2_);
                    splitTf32(xb.w, h3, l3_);
                    mmaTf32(sa[1], h0, h1, h2, h3, qh.z, qh.w);
                    mmaTf32(sb[1], l0_, l1_, l2_, l3_, qh.z, qh.w);
                    mmaTf32(sc[1], h0, h1, h2, h3, ql.z, ql.w);
                }
            }
        }
        __syncwarp();  // every lane has read its part of K
        requestK(i + SLOTS);
        auto dot = [&](int i) { return (sa[0][i] + sa[1][i]) + ((sb[0][i] + sb[1][i]) + (sc[0][i] + sc[1][i])); };
        const float s00 = tokA < len0 ? dot(0) * cs : -INFINITY;
        const float s01 = tokA < len1 ? dot(1) * cs : -INFINITY;
        const float s10 = tokB < len0 ? dot(2) * cs : -INFINITY;
        const float s11 = tokB < len1 ? dot(3) * cs : -INFINITY;
        float mx0 = fmaxf(s00, s10), mx1 = fmaxf(s01, s11);
#pragma unroll
        for (int off = 4; off <= 16; off <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
        }
        const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
        if (__any_sync(0xffffffffu, mn0 != m0 || mn1 != m1)) {
            const float a0 = fastExp2(m0 - mn0), a1 = fastExp2(m1 - mn1);
#pragma unroll
            for (int i = 0; i < MTO; ++i) {
                o[i][0] *= a0;
                o[i][1] *= a1;
                o[i][2] *= a0;
                o[i][3] *= a1;
            }
            l0 *= a0;
            l1 *= a1;
            m0 = mn0;
            m1 = mn1;
        }
        const float p00 = fastExp2(s00 - m0), p01 = fastExp2(s01 - m1);
        const float p10 = fastExp2(s10 - m0), p11 = fastExp2(s11 - m1);
        l0 += p00 + p10;
        l1 += p01 + p11;
        // rows past the chunk may hold anything (stale rows, other sequences): a 0
        // probability must not meet a NaN/Inf value, so those V rows are zeroed below
        // transpose p to the B layout through the warp's scratch: [token][column]
        *reinterpret_cast<float2 *>(pS + g * 8 + 2 * t) = make_float2(p00, p01);
        *reinterpret_cast<float2 *>(pS + (g + 8) * 8 + 2 * t) = make_float2(p10, p11);
        __syncwarp();
        uint32_t phi[2][2], plo[2][2];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            splitTf32(pS[(8 * kk + 2 * t) * 8 + g], phi[kk][0], plo[kk][0]);
            splitTf32(pS[(8 * kk + 2 * t + 1) * 8 + g], phi[kk][1], plo[kk][1]);
        }
        __syncwarp();
        // ---- O^T += V^T . P^T (HD dims x 8 columns), 3xTF32 ----
        cpAsyncWait<2 * SLOTS - 1>();  // V of this tile is in, the next K may still be on its way
        float own[kOwnSums ? MTO : 1][4];  // this tile's products
        if constexpr (kOwnSums) {
#pragma unroll
            for (int d = 0; d < MTO; ++d) own[d][0] = own[d][1] = own[d][2] = own[d][3] = 0.0f;
        }
        auto sum = [&](int d) -> float (&)[4] { return kOwnSums ? own[kOwnSums ? d : 0] : o[d]; };
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            const uint32_t ra = 8 * kk + 2 * t, rb = ra + 1;  // token rows of k slots t and t+4
            const bool okA = tok0 + ra < t1, okB = tok0 + rb < t1;
#pragma unroll
            for (int bx = 0; bx < NB; ++bx) {
                const uint8_t *vT = slotK(i) + L::kTileBytes + bx * T * 128;
                float4 xa = *reinterpret_cast<const float4 *>(vT + ra * 128 + ((g ^ (ra & 7u)) << 4));
                float4 xb = *reinterpret_cast<const float4 *>(vT + rb * 128 + ((g ^ (rb & 7u)) << 4));
                if (!okA) xa = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!okB) xb = make_float4(0.f, 0.f, 0.f, 0.f);
                {
                    uint32_t h0, l0_, h1, l1_, h2, l2_, h3, l3_;
                    splitTf32(xa.x, h0, l0_);
                    splitTf32(xa.y, h1, l1_);
                    splitTf32(xb.x, h2, l2_);
                    splitTf32(xb.y, h3, l3_);
                    mmaTf32(sum(2 * bx), h0, h1, h2, h3, phi[kk][0], phi[kk][1]);
                    mmaTf32(sum(2 * bx), l0_, l1_, l2_, l3_, phi[kk][0], phi[kk][1]);
                    mmaTf32(sum(2 * bx), h0, h1, h2, h3, plo[kk][0], plo[kk][1]);
                }
                {
                    uint32_t h0, l0_, h1, l1_, h2, l2_, h3, l3_;
                    splitTf32(xa.z, h0, l0_);
                    splitTf32(xa.w, h1, l1_);
                    splitTf32(xb.z, h2, l2_);
                    splitTf32(xb.w, h3, l3_);
                    mmaTf32(sum(2 * bx + 1), h0, h1, h2, h3, phi[kk][0], phi[kk][1]);
                    mmaTf32(sum(2 * bx + 1), l0_, l1_, l2_, l3_, phi[kk][0], phi[kk][1]);
                    mmaTf32(sum(2 * bx + 1), h0, h1, h2, h3, plo[kk][0], plo[kk][1]);
                }
            }
        }
        if constexpr (kOwnSums) {
#pragma unroll
            for (int d = 0; d < MTO; ++d)
#pragma unroll
                for (int k = 0; k < 4; ++k) o[d][k] += own[d][k];
        }
        __syncwarp();
        requestV(i + SLOTS);
    }

    // ---- fold the consumer warps, then the blocks of the cluster ----
#pragma unroll
    for (int off = 4; off <= 16; off <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, off);
        l1 += __shfl_xor_sync(0xffffffffu, l1, off);
    }
    namedBarSync(1, NW * 32);
    float *scr = reinterpret_cast<float *>(smem);
    using F = FoldScratch<HD>;
    constexpr int kWarpScr = F::kWarp;
    float *wO = scr + warp * kWarpScr;
#pragma unroll
    for (int bx = 0; bx < NB; ++bx) {
        const int d = 32 * bx + 4 * g;
        *reinterpret_cast<float4 *>(wO + (2 * t) * F::kRow + d) =
                make_float4(o[2 * bx][0], o[2 * bx][2], o[2 * bx + 1][0], o[2 * bx + 1][2]);
        *reinterpret_cast<float4 *>(wO + (2 * t + 1) * F::kRow + d) =
                make_float4(o[2 * bx][1], o[2 * bx][3], o[2 * bx + 1][1], o[2 * bx + 1][3]);
    }
    if (g == 0) {
        wO[F::kM + 2 * t] = m0;
        wO[F::kM + 2 * t + 1] = m1;
        wO[F::kL + 2 * t] = l0;
        wO[F::kL + 2 * t + 1] = l1;
    }
    namedBarSync(1, NW * 32);
    if (!ROWS) {
        FoldTarget f;
        f.out = p.out, f.pAcc = p.pAcc, f.pM = p.pM, f.pL = p.pL;
        f.numChunks = p.numChunks, f.slot = chunk / clusterSize();
        f.firstHead = static_cast<uint32_t>(colIndex(0)), f.nValid = min(8u, p.group - p.colBase);
        f.direct = p.directOut;
        f.qRot = p.tok.qRot != nullptr ? p.tok.qRot + colIndex(0) * HD : nullptr;
        f.cosT = p.tok.cosT, f.sinT = p.tok.sinT, f.tableRow = len - 1u;
        clusterFold<HD, NW>(scr, f, threadIdx.x);
        return;
    }
    constexpr int NV = HD / 4;  // float4 per output vector
    for (uint32_t idx = threadIdx.x; idx < 8 * NV; idx += NW * 32) {
        const uint32_t d4 = idx % NV, j = idx / NV;
        if (!colValid(j)) continue;
        float M = kNegBig;
#pragma unroll
        for (int w = 0; w < NW; ++w) M = fmaxf(M, scr[w * kWarpScr + F::kM + j]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float lsum = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const float *s = scr + w * kWarpScr;
            const float wgt = fastExp2(s[F::kM + j] - M);
            lsum += wgt * s[F::kL + j];
            const float4 a = *reinterpret_cast<const float4 *>(s + j * F::kRow + 4 * d4);
            acc.x = fmaf(wgt, a.x, acc.x);
            acc.y = fmaf(wgt, a.y, acc.y);
            acc.z = fmaf(wgt, a.z, acc.z);
            acc.w = fmaf(wgt, a.w, acc.w);
        }
        const float inv = lsum > 0.0f ? 1.0f / lsum : 0.0f;
        *reinterpret_cast<float4 *>(p.out + colIndex(j) * HD + 4 * d4) =
                make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    }
}

// Warps of the causal form: as many as the registers and the shared memory of an SM carry.
template <int HD>
struct KvShape {
    static constexpr int kRowsWarps = HD == 64 ? 16 : (HD == 128 ? 12 : 6);
};

template <int HD>
static int launchRows(const DecodeKvParams &prm, cudaStream_t st) {
    constexpr int NW = KvShape<HD>::kRowsWarps;
    using L = DecodeKvSmem<HD, NW, 1, false>;
    auto kern = decodeKvKernel<HD, NW, 1, 1, true>;
    static bool attrDone[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attrDone[dev]) {
        TC_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal));
        attrDone[dev] = true;
    }
    return launchDependent(kern, dim3(1, prm.nHeads, (prm.qRows + 7) / 8), NW * 32, L::kTotal, st, 1, prm);
}

static int kvCommonChecks(const char *who, const float *q, const void *kvK, const void *kvV, float *out,
                          uint32_t nHeads, uint32_t nKV, uint32_t hd, uint64_t totalRows, int kvHalf) {
    TC_REQUIRE(q && kvK && kvV && out, TC_EINVAL, "%s: null pointer", who);
    TC_REQUIRE(hd == 64 || hd == 128 || (hd == 256 && !kvHalf), TC_EUNSUPPORTED,
               "%s: head_dim %u (built for 64, 128 and -- f32 cache only -- 256)", who, hd);
    TC_REQUIRE(nKV > 0 && nHeads % nKV == 0, TC_EINVAL, "%s: nHeads %u not a multiple of nKV %u", who, nHeads, nKV);
    TC_REQUIRE(nHeads / nKV <= 64, TC_EUNSUPPORTED, "%s: %u q heads per kv head (built for <= 64)", who, nHeads / nKV);
    TC_REQUIRE(totalRows >= 1 && totalRows < (1ull << 31), TC_EUNSUPPORTED, "%s: cache of %llu rows", who,
               (unsigned long long) totalRows);
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(kvK) | reinterpret_cast<uintptr_t>(kvV) | reinterpret_cast<uintptr_t>(q) |
                 reinterpret_cast<uintptr_t>(out)) & 15u) == 0,
               TC_EINVAL, "%s: q/out/K/V need 16-byte alignment", who);
    return TC_OK;
}

// rows mode: causal attention of seqLen query rows (row s sees [0, cachePos + s])
static int prefillKv(const float *q, const void *kvK, const void *kvV, float *out, uint32_t seqLen, uint32_t nHeads,
                     uint32_t nKV, uint32_t hd, uint32_t cachePos, const uint32_t *devPos, uint64_t totalRows,
                     float invSqrt, int kvHalf, cudaStream_t st) {
    int rc = kvCommonChecks("prefill_kv", q, kvK, kvV, out, nHeads, nKV, hd, totalRows, kvHalf);
    if (rc != TC_OK) return rc;
    if (seqLen == 0) return TC_OK;
    if (devPos == nullptr && static_cast<uint64_t>(cachePos) + seqLen > totalRows) {
        setError("prefill_kv: rows [%u, %llu) pass the cache of %llu rows", cachePos,
                 (unsigned long long) cachePos + seqLen, (unsigned long long) totalRows);
        return TC_ECONTEXT_FULL;
    }
    const uint32_t rowBlocks = (seqLen + 7) / 8;
    TC_REQUIRE(rowBlocks <= 65535 && nHeads <= 65535, TC_EUNSUPPORTED, "prefill_kv: %u rows x %u heads", seqLen, nHeads);
    // (a position on the device: somewhere in the store)
    const uint64_t before = devPos == nullptr ? cachePos : (totalRows > seqLen ? (totalRows - seqLen) / 2 : 0);
    if (prefillExactWins(seqLen, before, nHeads, hd, kvHalf))
        return prefillExact(q, kvK, kvV, out, seqLen, nHeads, nKV, hd, cachePos, devPos, totalRows, invSqrt, kvHalf, st);
    DecodeKvParams prm;
    memset(&prm, 0, sizeof(prm));
    prm.q = q;
    prm.out = out;
    prm.devPos = devPos;
    prm.totalRows = totalRows;
    prm.nHeads = nHeads;
    prm.nKV = nKV;
    prm.group = nHeads / nKV;
    prm.numChunks = 1;
    prm.kvK = const_cast<void *>(kvK), prm.kvV = const_cast<void *>(kvV);
    prm.qRows = seqLen;
    prm.cachePos = cachePos;
    prm.invSqrt = invSqrt;
    prm.directOut = 1;
    prm.err = devErrorWord();
    TC_REQUIRE(prm.err != nullptr, TC_ECUDA, "prefill_kv: no device error word");
    if (kvHalf) return prefillKv16(prm, hd, st);
    if (hd == 64) return launchRows<64>(prm, st);
    if (hd == 256) return launchRows<256>(prm, st);
    return launchRows<128>(prm, st);
}

template <int HD, int NW, int SLOTS, int BPS>
static int decodeKv32(const DecodeKvParams &prm, uint8_t *q81Out, cudaStream_t st) {
    using L = DecodeKvSmem<HD, NW, SLOTS, kvSharesQuery(HD, BPS, false)>;
    static ClusterSetup setup;
    return launchKvDecode(setup, decodeKvKernel<HD, NW, SLOTS, BPS, false>, NW * 32, L::kTotal, HD, NW, 2 * L::kTileBytes,
                          HD == 256 ? 3.4f : (HD == 128 ? 2.85f : 1.7f), HD == 256 ? 0.8f : (HD == 128 ? 0.38f : 0.2f), prm,
                          q81Out, st);
}

int decodeKvToken(const float *q, const void *kvK, const void *kvV, float *attnOut, float *pAcc, float *pM, float *pL,
                  uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t pos, const uint32_t *devPos, uint64_t totalRows,
                  uint32_t numChunks, float invSqrt, int kvHalf, uint8_t *q81Out, const NewToken &tok, cudaStream_t st) {
    int rc = kvCommonChecks("tc_attn_decode_kv", q, kvK, kvV, attnOut, nHeads, nKV, hd, totalRows, kvHalf);
    if (rc != TC_OK) return rc;
    TC_REQUIRE(static_cast<uint64_t>(pos) + 1 <= totalRows, TC_ECONTEXT_FULL,
               "tc_attn_decode_kv: position %u is outside the cache of %llu rows", pos,
               (unsigned long long) totalRows);
    TC_REQUIRE(numChunks >= 1, TC_EWORKSPACE, "tc_attn_decode_kv: no chunk slots");
    DecodeKvParams prm;
    memset(&prm, 0, sizeof(prm));
    prm.q = q;
    prm.out = attnOut;
    prm.pAcc = pAcc;
    prm.pM = pM;
    prm.pL = pL;
    prm.devPos = devPos;
    prm.totalRows = totalRows;
    prm.lenHost = pos + 1;
    prm.nHeads = nHeads;
    prm.nKV = nKV;
    prm.group = nHeads / nKV;
    prm.numChunks = numChunks;
    prm.invSqrt = invSqrt;
    prm.tok = tok;
    prm.kvHalf = kvHalf != 0;
    prm.kvK = const_cast<void *>(kvK), prm.kvV = const_cast<void *>(kvV);
    prm.err = devErrorWord();
    TC_REQUIRE(prm.err != nullptr, TC_ECUDA, "tc_attn_decode_kv: no device error word");
    if (kvHalf) return decodeKv16(prm, hd, q81Out, st);
    // Warps of a block, slots of a warp, blocks per SM.  Rows that a 16-block cluster covers with one tile per warp (head_dim
    // 128: 1536) want small blocks; longer ones as many warps per SM as fit (head_dim 128, per layer: 2048 rows 8.6 against
    // 9.5 us, 20000 rows 23.8 against 26.4, 200 rows 7.2 against 6.5; head_dim 256, 16 / 4 heads with norm and gate: four warps 12.4 /
    // 32.4 / 43.1 us at 500 / 8191 / 12000 rows, six 11.9 / 29.0 / 34.6).
    if (hd == 64) return decodeKv32<64, 8, 2, 1>(prm, q81Out, st);
    if (hd == 128)
        return prm.lenHost <= 1536u ? decodeKv32<128, 6, 1, 2>(prm, q81Out, st) : decodeKv32<128, 8, 1, 1>(prm, q81Out, st);
    return decodeKv32<256, 6, 1, 1>(prm, q81Out, st);
}

}  // namespace tc

extern "C" {

int tc_attn_prefill_kv(const float *q, const void *kvK, const void *kvV, float *out, uint32_t seqLen,
                       uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t cachePos, const uint32_t *devPos,
                       uint64_t totalRows, float invSqrt, int kvHalf, tc_stream stream) {
    return tc::prefillKv(q, kvK, kvV, out, seqLen, nHeads, nKV, hd, cachePos, devPos, totalRows, invSqrt, kvHalf,
                         static_cast<cudaStream_t>(stream));
}

int tc_attn_decode_kv(const float *q, const void *kvK, const void *kvV, float *attnOut, float *pAcc, float *pM,
                      float *pL, uint32_t seqLen, uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t pos,
                      const uint32_t *devPos, uint64_t totalRows, uint32_t numChunks, uint32_t chunkSize,
                      float invSqrt, int kvHalf, uint8_t *q81Out, tc_stream stream) {
    (void) chunkSize;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (seqLen != 1) {
        // the reference only splits single-token decode; several rows take the causal kernel
        TC_REQUIRE(q81Out == nullptr, TC_EUNSUPPORTED, "tc_attn_decode_kv: Q8_1 output needs seqLen == 1");
        return tc::prefillKv(q, kvK, kvV, attnOut, seqLen, nHeads, nKV, hd, pos, devPos, totalRows, invSqrt, kvHalf, st);
    }
    tc::NewToken none;
    memset(&none, 0, sizeof(none));
    return tc::decodeKvToken(q, kvK, kvV, attnOut, pAcc, pM, pL, nHeads, nKV, hd, pos, devPos, totalRows, numChunks, invSqrt,
                             kvHalf, q81Out, none, st);
}

}  // extern "C"
