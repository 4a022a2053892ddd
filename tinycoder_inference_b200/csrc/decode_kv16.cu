// decode_kv16.cu -- grouped-query attention over an fp16 KV cache: split-KV decode and,
// with query rows as columns, the unsplit causal kernel.
//
// What it replaces: the KVT = __half instantiations of kWarpAttentionSplit /
// kWarpAttention(Pos) behind launchDecodeAttentionSplit(..., kvHalf = true, ...)
// (include/gpu/GpuAttentionKernels.hpp:211-272, 537-599, 625-766, 1129-1230), i.e. the
// dense models' optional fp16 cache (src/cpp/core/cuda/forward/GPUComputeUpload.cu:1252):
// score = dot(q, float(k)) * invSqrt, online softmax with exp2, out = sum p float(v) / sum p.
//
// Same skeleton as the f32 kernel (decode_kv.cu) -- a block streams a token range of one kv head,
// its warps take 16-token tiles in turn and serve every q head of the kv head, decode_cluster.cuh
// around it -- with the natural operands: fp16 K and V go into mma.sync.m16n8k16 as they are (ldmatrix for K,
// ldmatrix.trans for V, both straight from the tiles that each warp copies for itself, 128-byte swizzled), q and p are
// carried as fp16 hi + lo pairs (two MMAs, ~22 mantissa bits) after a power-of-two
// normalisation of q, accumulation is f32.  Nothing is rounded that the reference does not
// round: float(k) and float(v) are exact.  (A tensor-core product drops the bits of its running sum that do not fit, and
// those losses add up over a warp's tiles, hence the sums per tile; the small terms go first.  28 / 4 / 128, distance from
// a 64-bit evaluation with one sum throughout -> like this: 8191 rows 4.2e-7 -> 3.2e-7, 40000 rows 7.9e-7 -> 3.4e-7, for
// 7.71 -> 7.87 and 20.8 -> 21.0 us; the additions put off until the next tile's scores are under way: 7.93.)
#include "decode_cluster.cuh"

namespace tc {

// Every warp has SLOTS slots for 16-token tiles of K and as many of V, each as HD / 64 half-tiles of [16 rows][64 halves =
// 128 bytes], half-tile a covering dims [64a, 64a + 64).
template <int HD, int NW, int SLOTS, bool ROWS>
struct DecodeKv16Smem {
    static constexpr int kAtomBytes = 16 * 128;      // one half-tile
    static constexpr int kTileBytes = 16 * HD * 2;
    static constexpr int kSlots = NW * SLOTS * 2 * kTileBytes, kScratch = NW * FoldScratch<HD>::kWarp * 4;  // (the fold reuses the slots)
    static constexpr int kQuery = kSlots > kScratch ? kSlots : kScratch;   // decode: the block's query operands
    static constexpr int kTotal = kQuery + (ROWS ? 0 : HD * 32 + 32) + 128;
    static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

constexpr float kLazyLog2Kv16 = 8.0f;  // see decode_i8.cu: p stays <= 2^8, exact enough as fp16 hi + lo

// ROWS: the causal kernel (one block per 8 query rows and q head); otherwise decode, blocks of a cluster
// share a kv head's tokens.
template <int HD, int NW, int SLOTS, int BPS, bool ROWS>
__global__ void __launch_bounds__(NW * 32, BPS) decodeKv16Kernel(const __grid_constant__ DecodeKvParams p) {
    using L = DecodeKv16Smem<HD, NW, SLOTS, ROWS>;
    constexpr int T = 16;
    constexpr int NS = HD / 16;     // k16 steps of QK^T = 16-dim output tiles of PV

    const uint32_t chunk = blockIdx.x, hg = blockIdx.y, b = ROWS ? gridDim.z - 1u - blockIdx.z : blockIdx.z;  // (late rows first)
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;

    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 127) & ~uintptr_t(127));

    if (!ROWS) {
        // (a device position read here may be a step old: good enough to know which rows to pull)
        const uint32_t hint = p.devPos ? min(p.devPos[0], p.lenHost - 1u) + 1u : p.lenHost;
        const uint32_t per = p.devPos ? tokensPerBlock(hint, gridDim.x) : p.chunkTokens;
        const uint8_t *k = static_cast<const uint8_t *>(p.kvK) + static_cast<size_t>(hg) * HD * 2;
        const uint8_t *v = static_cast<const uint8_t *>(p.kvV) + static_cast<size_t>(hg) * HD * 2;
        for (uint32_t i = 0, tok = chunk * per + warp * T; i < kPrefetchTiles && tok < min(hint, (chunk + 1u) * per); ++i, tok += NW * T)
            prefetchTile<HD * 2>(k, v, static_cast<size_t>(p.nKV) * HD * 2, tok, p.totalRows - 1, lane);
        const size_t row = static_cast<size_t>(hg) * HD, table = static_cast<size_t>(p.lenHost - 1u) * (HD / 2);
        const bool rotates = p.tok.cosT != nullptr && p.devPos == nullptr;
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
    const uint32_t stride = p.nKV * HD * 2;
    const uint8_t *storeK = static_cast<const uint8_t *>(p.kvK) + static_cast<size_t>(kvHead) * HD * 2;
    const uint8_t *storeV = static_cast<const uint8_t *>(p.kvV) + static_cast<size_t>(kvHead) * HD * 2;
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
            copyTile<T, HD * 2>(smemAddr(slotK(i) + (isV ? L::kTileBytes : 0)), isV ? storeV : storeK, stride, row,
                                have > row ? have - row : 0u, lane);
        cpAsyncCommit();
    };
    auto requestK = [&](uint32_t i) { request(i, false); };
    auto requestV = [&](uint32_t i) { request(i, true); };
    NewRow<HD> fresh;
    // (behind the loads of q, which would queue behind the tiles' otherwise: 28 / 4 / 128 at 8191 / 20000 rows 8.6 / 13.6 -> 7.5 / 13.0 us
    // a layer, 8 / 4 / 64 at 2000 / 20000 rows 4.7 / 10.0 -> 4.5 / 9.1)
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

    // q of column n = g as the B operand of k16 step s: b0 = dims 16s + 2t, +1; b1 = dims
    // 16s + 8 + 2t, +1.  Power-of-two normalised, split into fp16 hi + lo.
    uint32_t qhi[NS][2], qlo[NS][2];
    float cs0, cs1;
    auto exponent = [](float amax) {
        const int e = static_cast<int>((__float_as_uint(amax) >> 23) & 0xffu) - 127;  // floor(log2 amax)
        return amax > 0.0f ? max(-100, min(100, e)) : 0;
    };
    if constexpr (ROWS) {
        const bool valid = colValid(g);
        const float *qp = p.q + colIndex(valid ? g : 0) * HD;
        float2 qv[NS][2];
        float amax = 0.0f;
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                qv[s][h] = valid ? *reinterpret_cast<const float2 *>(qp + 16 * s + 8 * h + 2 * t)
                                 : make_float2(0.f, 0.f);
            }
        requestFirst();
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h) amax = fmaxf(amax, fmaxf(fabsf(qv[s][h].x), fabsf(qv[s][h].y)));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const int e = exponent(amax);
        const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);  // 2^-e
        const float up = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);    // 2^e
        const float headScale = p.invSqrt * up * kLog2e;
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float h0, l0, h1, l1;
                splitHalf(qv[s][h].x * down, h0, l0);
                splitHalf(qv[s][h].y * down, h1, l1);
                qhi[s][h] = packHalf2(h0, h1);
                qlo[s][h] = packHalf2(l0, l1);
            }
        cs0 = __shfl_sync(0xffffffffu, headScale, (2 * t) * 4);
        cs1 = __shfl_sync(0xffffffffu, headScale, (2 * t + 1) * 4);
    } else {
        // The block's warps share the work, a column at a time each: a lane takes dims 2 lane, + 1 of both halves of the
        // vector (partners of the NEOX rotation) and leaves them where the operands are read.  (Every warp for itself took 350
        // instructions.  Per layer, before -> with this: 28 / 4 / 128 at 500 / 2000 / 8191 rows 5.05 / 5.9 / 9.45 -> 4.45 / 5.2 / 8.55
        // us, 14 / 2 / 64 at 2000 rows 4.7 -> 4.5; 8 / 4 / 64 at 20 rows 3.3 -> 3.4.)
        uint32_t *frag = reinterpret_cast<uint32_t *>(smem + L::kQuery);  // [step][lane]: hi 0, hi 1, lo 0, lo 1
        float *scale = reinterpret_cast<float *>(smem + L::kQuery + HD * 32);
        static_assert(ROWS || NW == 8, "a column per warp");
        {
            const uint32_t j = warp;
            const bool valid = colValid(j) && 2 * lane < HD / 2, rotate = valid && p.tok.cosT != nullptr;
            // (plain loads: with a rotation q is written in place at the end of the launch)
            float2 x = make_float2(0.f, 0.f), y = x, c = x, sn = x;
            if (valid) {
                const float *qp = p.q + colIndex(j) * HD + 2 * lane;
                x = *reinterpret_cast<const float2 *>(qp), y = *reinterpret_cast<const float2 *>(qp + HD / 2);
            }
            if (rotate) {
                const size_t at = static_cast<size_t>(len - 1u) * (HD / 2) + 2 * lane;
                c = *reinterpret_cast<const float2 *>(p.tok.cosT + at), sn = *reinterpret_cast<const float2 *>(p.tok.sinT + at);
            }
            requestFirst();
            if (rotate) {
                const float2 x0 = x, x1 = y;
                x = make_float2(fmaf(x0.x, c.x, -__fmul_rn(x1.x, sn.x)), fmaf(x0.y, c.y, -__fmul_rn(x1.y, sn.y)));
                y = make_float2(fmaf(x0.x, sn.x, __fmul_rn(x1.x, c.x)), fmaf(x0.y, sn.y, __fmul_rn(x1.y, c.y)));
            }
            const float top = fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(y.x), fabsf(y.y)));
            // (maxima of non-negative floats, by their bits)
            const int e = exponent(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(top))));
            const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);  // 2^-e
            if (lane == 0) scale[j] = p.invSqrt * __uint_as_float(static_cast<uint32_t>(127 + e) << 23) * kLog2e;
            if (2 * lane < HD / 2) {
#pragma unroll
                for (uint32_t half = 0; half < 2; ++half) {
                    const float2 v = half ? y : x;
                    const uint32_t dim = half * (HD / 2) + 2 * lane;
                    uint32_t *to = frag + ((dim / 16) * 32 + j * 4 + (dim % 8) / 2) * 4 + (dim % 16) / 8;
                    float h0, l0, h1, l1;
                    splitHalf(v.x * down, h0, l0);
                    splitHalf(v.y * down, h1, l1);
                    to[0] = packHalf2(h0, h1);
                    to[2] = packHalf2(l0, l1);
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const uint4 f = *reinterpret_cast<const uint4 *>(frag + (s * 32 + lane) * 4);
            qhi[s][0] = f.x, qhi[s][1] = f.y, qlo[s][0] = f.z, qlo[s][1] = f.w;
        }
        cs0 = scale[2 * t], cs1 = scale[2 * t + 1];
    }
    const uint32_t len0 = colLen(2 * t), len1 = colLen(2 * t + 1);

    if (mine) {
        const size_t at = (static_cast<size_t>(len - 1u) * p.nKV + kvHead) * HD;
        uint8_t *tile = intoTile ? slotK((nTiles - 1u) / NW) : nullptr;
        fresh.store(p.tok.cosT != nullptr, static_cast<__half *>(p.kvK) + at, static_cast<__half *>(p.kvV) + at, tile,
                    tile + L::kTileBytes, len - 1u - (t0 + (nTiles - 1u) * T), lane);
        __syncwarp();
    }

    float m0 = kNegBig, m1 = kNegBig, l0 = 0.0f, l1 = 0.0f;
    float o[NS][4];
#pragma unroll
    for (int i = 0; i < NS; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    // Where a warp takes several tiles (SLOTS > 1), a tile's products have sums of their own: see the head of the file.
    constexpr bool kOwnSums = SLOTS > 1;

    const uint32_t lr = (lane & 7u) + ((lane >> 3) & 1u) * 8u;  // ldmatrix row this lane addresses
    const uint32_t lco = lane >> 4;                             // and which 16-byte chunk of the pair
    const uint32_t lmOff = lr * 128;

    for (uint32_t i = 0, tile = warp; tile < nTiles; ++i, tile += NW) {
        cpAsyncWait<2 * SLOTS - 1>();  // K of this tile is in, V may still be on its way
        const uint32_t tokW = t0 + tile * T;  // first token of the tile
        const uint32_t tokA = tokW + g, tokB = tokA + 8;

        // ---- S^T = K . Q^T (16 tokens x 8 columns) ----
        float sh[4] = {0.f, 0.f, 0.f, 0.f}, sl[4] = {0.f, 0.f, 0.f, 0.f};
        const uint32_t kTile = smemAddr(slotK(i));
#pragma unroll
        for (int ks = 0; ks < NS; ++ks) {
            const uint32_t sw = (((2 * (ks & 3) + lco) ^ (lr & 7u)) << 4) + (ks >> 2) * L::kAtomBytes;
            uint32_t r0, r1, r2, r3;  // rows 0-7 / 8-15 of dims 16ks..+7, then of dims 16ks+8..+15
            ldmatrixX4(r0, r1, r2, r3, kTile + lmOff + sw);
            mmaF16(sh, r0, r1, r2, r3, qhi[ks][0], qhi[ks][1]);
            mmaF16(sl, r0, r1, r2, r3, qlo[ks][0], qlo[ks][1]);
        }
        __syncwarp();  // every lane has read its part of K
        requestK(i + SLOTS);
        // a stale or foreign row behind the range may hold anything, NaN included: select, never scale
        const float s00 = tokA < len0 ? (sh[0] + sl[0]) * cs0 : -INFINITY;
        const float s01 = tokA < len1 ? (sh[1] + sl[1]) * cs1 : -INFINITY;
        const float s10 = tokB < len0 ? (sh[2] + sl[2]) * cs0 : -INFINITY;
        const float s11 = tokB < len1 ? (sh[3] + sl[3]) * cs1 : -INFINITY;
        float mx0 = fmaxf(s00, s10), mx1 = fmaxf(s01, s11);
#pragma unroll
        for (int off = 4; off <= 16; off <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
        }
        const float mn0 = mx0 > m0 + kLazyLog2Kv16 ? mx0 : m0;
        const float mn1 = mx1 > m1 + kLazyLog2Kv16 ? mx1 : m1;
        if (__any_sync(0xffffffffu, mn0 != m0 || mn1 != m1)) {
            const float a0 = fastExp2(m0 - mn0), a1 = fastExp2(m1 - mn1);
#pragma unroll
            for (int i = 0; i < NS; ++i) {
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
        // p as fp16 hi + lo, transposed to the B layout (tokens 2t, 2t+1 / 8+2t, 8+2t+1 of column g)
        uint32_t bh[2], bl[2];
        {
            const float p00 = fastExp2(s00 - m0), p01 = fastExp2(s01 - m1);
            const float p10 = fastExp2(s10 - m0), p11 = fastExp2(s11 - m1);
            l0 += p00 + p10;
            l1 += p01 + p11;
            float h0, q0, h1, q1;
            splitHalf(p00, h0, q0);
            splitHalf(p01, h1, q1);
            bh[0] = movmatrixTrans(packHalf2(h0, h1));
            bl[0] = movmatrixTrans(packHalf2(q0, q1));
            splitHalf(p10, h0, q0);
            splitHalf(p11, h1, q1);
            bh[1] = movmatrixTrans(packHalf2(h0, h1));
            bl[1] = movmatrixTrans(packHalf2(q0, q1));
        }
        // ---- O^T += V^T . P^T (HD dims x 8 columns), V read transposed ----
        // rows behind the chunk get probability 0, but 0 * NaN is NaN: clear those V rows.
        // Register halves of a transposed fragment are tokens 2t (low) and 2t+1 (high).
        uint32_t mk0 = 0xffffffffu, mk1 = 0xffffffffu;
        if (tokW + 16 > t1) {
            mk0 = (tokW + 2 * t < t1 ? 0x0000ffffu : 0u) | (tokW + 2 * t + 1 < t1 ? 0xffff0000u : 0u);
            mk1 = (tokW + 8 + 2 * t < t1 ? 0x0000ffffu : 0u) | (tokW + 8 + 2 * t + 1 < t1 ? 0xffff0000u : 0u);
        }
        cpAsyncWait<2 * SLOTS - 1>();  // V of this tile is in, the next K may still be on its way
        const uint32_t vTile = smemAddr(slotK(i) + L::kTileBytes);
#pragma unroll
        for (int ks = 0; ks < NS; ++ks) {
            const uint32_t sw = (((2 * (ks & 3) + lco) ^ (lr & 7u)) << 4) + (ks >> 2) * L::kAtomBytes;
            uint32_t r0, r1, r2, r3;  // (tokens 0-7, dims lo) (tokens 8-15, dims lo) (0-7, dims hi) (8-15, dims hi)
            ldmatrixX4Trans(r0, r1, r2, r3, vTile + lmOff + sw);
            r0 &= mk0;
            r2 &= mk0;
            r1 &= mk1;
            r3 &= mk1;
            // A rows g / g+8 = dims 16ks + g / + 8 + g; k = tokens
            float own[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            float(&sum)[4] = kOwnSums ? own : o[ks];
            mmaF16(sum, r0, r2, r1, r3, bl[0], bl[1]);
            mmaF16(sum, r0, r2, r1, r3, bh[0], bh[1]);
            if (kOwnSums) {
#pragma unroll
                for (int i = 0; i < 4; ++i) o[ks][i] += own[i];
            }
        }
        __syncwarp();
        requestV(i + SLOTS);
    }

    // ---- fold the consumer warps of each kv head, write the chunk partial ----
#pragma unroll
    for (int off = 4; off <= 16; off <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, off);
        l1 += __shfl_xor_sync(0xffffffffu, l1, off);
    }
    namedBarSync(1, NW * 32);  // every consumer is done reading the ring
    float *scr = reinterpret_cast<float *>(smem);
    using F = FoldScratch<HD>;
    constexpr int kWarpScr = F::kWarp;
    float *wO = scr + warp * kWarpScr;  // [8 columns][FoldScratch::kRow], then m[8], l[8]
#pragma unroll
    for (int c = 0; c < NS; ++c) {
        const int d = 16 * c + g;
        wO[(2 * t) * F::kRow + d] = o[c][0];
        wO[(2 * t + 1) * F::kRow + d] = o[c][1];
        wO[(2 * t) * F::kRow + d + 8] = o[c][2];
        wO[(2 * t + 1) * F::kRow + d + 8] = o[c][3];
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

template <int HD, int NW, int SLOTS, int BPS>
static int decodeKv16Hd(const DecodeKvParams &prm, uint8_t *q81Out, cudaStream_t st) {
    using L = DecodeKv16Smem<HD, NW, SLOTS, false>;
    static ClusterSetup setup;
    // (head_dim 64, 0.73 -> 0.61 with two slots: 14 / 2 at 9000 rows 27.2 -> 24.8 us for four layers, 8 / 4 at 12000 33.5 -> 27.7; with
    // four slots 14 / 2 at 45000 rows 18.6 -> 19.3 for two)
    return launchKvDecode(setup, decodeKv16Kernel<HD, NW, SLOTS, BPS, false>, NW * 32, L::kTotal, HD, NW, 2 * L::kTileBytes,
                          HD == 128 ? 0.87f : SLOTS == 4 ? 0.73f : 0.61f, HD == 128 ? 0.12f : 0.08f, prm, q81Out, st);
}

// Both are called from decode_kv.cu when kvHalf is set; arguments were validated there.
// Warps of a block, slots of a warp, blocks per SM: rows beyond what a 16-block cluster covers with one tile per warp
// (2048) want two tiles of a warp in flight (head_dim 128, per layer: 20000 rows 14.3 against 15.8 us, 47000 rows 24.2
// against 28.3; 2047 rows 6.0 against 5.9).  Half as wide rows beyond what a cluster covers alone want four of them
// (14 / 2 / 64: 20000 rows 8.2 -> 7.8 us, 47000 10.7 -> 10.1; 12000 rows 6.8 -> 6.9).
int decodeKv16(const DecodeKvParams &prm, uint32_t hd, uint8_t *q81Out, cudaStream_t st) {
    if (hd == 64)
        return prm.lenHost <= 2048u    ? decodeKv16Hd<64, 8, 1, 2>(prm, q81Out, st)
               : prm.lenHost <= 16384u ? decodeKv16Hd<64, 8, 2, 1>(prm, q81Out, st)
                                       : decodeKv16Hd<64, 8, 4, 1>(prm, q81Out, st);
    return prm.lenHost <= 2048u ? decodeKv16Hd<128, 8, 1, 2>(prm, q81Out, st) : decodeKv16Hd<128, 8, 2, 1>(prm, q81Out, st);
}

template <int HD>
static int rowsKv16Hd(const DecodeKvParams &prm, cudaStream_t st) {
    constexpr int NW = 16;
    using L = DecodeKv16Smem<HD, NW, 1, true>;
    auto kern = decodeKv16Kernel<HD, NW, 1, 1, true>;
    static bool attrDone[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attrDone[dev]) {
        TC_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal));
        attrDone[dev] = true;
    }
    return launchDependent(kern, dim3(1, prm.nHeads, (prm.qRows + 7) / 8), NW * 32, L::kTotal, st, 1, prm);
}

int prefillKv16(DecodeKvParams prm, uint32_t hd, cudaStream_t st) {
    return hd == 64 ? rowsKv16Hd<64>(prm, st) : rowsKv16Hd<128>(prm, st);
}

}  // namespace tc
