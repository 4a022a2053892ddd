// decode_i8.cu -- grouped-query decode attention over the int8 KV store.
//
// What it replaces: kQ35WarpAttention8Split + kAttnCombinePartial and the eager
// kQ35WarpAttention8 of the reference (include/gpu/GpuQwen35Kernels.hpp:519-581,
// 641-692): q f32 [nHeads][hd], K/V rows int8 with one f32 scale per (row, kv
// head), score = dot(q, float(k8)*sk) * invSqrt, online softmax with exp2,
// out = sum p * float(v8)*sv / sum p.
//
// This file: the mma.sync form, for head_dim 256 and for causal query rows over the store (head_dim 128 decode is
// decode_i8_tc.cu's), and the entry points of both.
//   * decode: a block streams a token range of one kv head and serves ALL its q heads, so every KV byte leaves
//     HBM exactly once; the split over clusters of blocks and the fold of their results are decode_cluster.cuh's,
//     and the launch quantises the new token's row itself.
//   * the warps of a block take tiles of MT x 16 tokens in turn, each with copies (16-byte cp.async) and slots of its
//     own: a warp spends a microsecond on 16 tokens, HBM half of that for an SM, so it takes many independent warps.
//   * at group 5..8 the dequant+FMA work (2*group flop per KV byte) is beyond the CUDA cores at HBM speed, so
//     QK^T and PV run on tensor cores (mma.sync.m16n8k16): int8 is fed as exact fp16 subnormals, q and p*sv are
//     carried as fp16 hi+lo pairs (two MMAs, ~22 mantissa bits) after a power-of-two normalisation, accumulation
//     is f32.  The per-row K scale is applied to the score column after the MMA, the V scale is folded into p
//     before it.
//   * S is produced transposed (tokens x heads) so no MMA row is padding; the probabilities reach the PV operand
//     layout through movmatrix.trans.
#include <mutex>

#include "decode_i8.cuh"

namespace tc {

constexpr int kHD = 128;

// MT = 16-row MMA tiles a consumer warp folds at a time: 2 amortises the softmax bookkeeping over 32
// tokens (causal rows at head_dim 128).
//
// Every warp has NS slots for tiles of 16 MT tokens of K and as many of V, each as HD/128 half-tiles of [rows][128 bytes],
// half-tile h covering dims [128h, 128h + 128); the rows' scales lie behind all slots.
template <int HD, int NW, int NS, int MT, bool ROWS>
struct DecodeI8Smem {
    static constexpr int T = 16 * MT;
    static constexpr int kHalfBytes = T * 128;            // one half-tile
    static constexpr int kTileBytes = T * HD;             // K (or V) bytes of a tile
    static constexpr int kScales = NW * NS * 2 * kTileBytes;   // [warp][slot][K, V][T] floats
    static constexpr int kSlots = kScales + NW * NS * 2 * T * 4, kScratch = NW * FoldScratch<HD>::kWarp * 4;  // (the fold reuses the slots)
    static constexpr int kQuery = kSlots > kScratch ? kSlots : kScratch;   // decode: the block's query fragments
    static constexpr int kTotal = kQuery + (ROWS ? 0 : I8QueryShare<HD, NW>::kBytes) + 128;
    static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

// ROWS: causal query rows; otherwise a token's q heads over chunks of the store: SW warps share a chunk, a block holds NW / SW
// neighbouring chunks.
template <int HD, int NW, int SW, int NS, int MT, bool ROWS>
__global__ void __launch_bounds__(NW * 32, 1)
decodeI8Kernel(const __grid_constant__ DecodeI8Params p) {
    using L = DecodeI8Smem<HD, NW, NS, MT, ROWS>;
    static_assert(!ROWS || SW == NW, "rows share all tiles");
    constexpr int T = L::T;
    constexpr int NC = HD / 16;  // 16-dim groups of a head vector
    constexpr int NR = 2 * MT;  // 8-token row groups of a warp's tile
    constexpr float k2p24 = kI8Unscale;

    constexpr uint32_t G = NW / SW;  // chunks of a block
    const uint32_t hg = blockIdx.y, b = ROWS ? gridDim.z - 1u - blockIdx.z : blockIdx.z;  // (late rows first)
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t chunk = blockIdx.x * G + warp / SW, sw = warp % SW;

    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 127) & ~uintptr_t(127));

    if (!ROWS && p.devLens == nullptr && p.devRowBase == nullptr) {
        const uint64_t base = static_cast<uint64_t>(b) * p.rowsPerSeq;
        const uint32_t t0 = chunk * p.chunkTokens, t1 = min(p.lenHost, t0 + p.chunkTokens);
        const uint8_t *k = reinterpret_cast<const uint8_t *>(p.k8w) + static_cast<size_t>(hg) * HD;
        const uint8_t *v = reinterpret_cast<const uint8_t *>(p.v8w) + static_cast<size_t>(hg) * HD;
        for (uint32_t i = 0, tok = t0 + sw * T; i < kPrefetchTiles && tok < t1; ++i, tok += SW * T) {
            prefetchTile<HD>(k, v, static_cast<size_t>(p.nKV) * HD, base + tok, p.totalRows - 1, lane);
            if (lane < 2u) {
                const float *s = (lane ? p.vs : p.ks) + min(base + tok, p.totalRows - 1) * p.nKV + hg;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(s));
            }
        }
    }
    if (!ROWS) {
        const size_t row = (static_cast<size_t>(b) * p.nKV + hg) * HD;
        prefetchToken<HD>(p.q + (static_cast<size_t>(b) * p.nHeads + hg * p.group + p.colBase) * HD, min(8u, p.group - p.colBase),
                          p.appendK != nullptr ? p.appendK + row : nullptr, p.appendV + row, nullptr, nullptr, threadIdx.x);
    }
    gridDepWait();
    gridDepLaunch();

    uint32_t len, rowsPos = p.cachePos;  // rows mode: first query row sits at pool row rowsPos
    if (ROWS) {
        if (p.devPos) rowsPos = p.devPos[0];
        len = rowsPos + min(p.qRows, b * 8u + 8u);  // b = row block; its last row sees [0, len)
    } else {
        // (the host's length is the upper bound of a device length)
        len = p.devLens ? min(p.devLens[b] + p.lenAdd, p.lenHost) : p.lenHost;
        // a cluster behind the last row leaves as a whole: the merge derives the active count from len.  The first one stays: it
        // writes the zeros of a sequence without rows
        if ((blockIdx.x - clusterRank()) * G * p.chunkTokens >= len && blockIdx.x != clusterRank()) return;
    }
    const uint32_t t0 = ROWS ? 0u : chunk * p.chunkTokens;
    if (!ROWS && clusterSize() > 1) clusterHello();
    const uint32_t t1 = ROWS ? len : min(len, t0 + p.chunkTokens);
    const uint32_t nTiles = t0 < t1 ? (t1 - t0 + T - 1) / T : 0u;
    const uint64_t rowBase = ROWS ? 0ull : (p.devRowBase ? p.devRowBase[b] : static_cast<uint64_t>(b) * p.rowsPerSeq);
    const uint32_t kvHead = ROWS ? hg / p.group : hg;

    // Tile j of a chunk belongs to its warp j % SW, slot (j / SW) % NS.  A warp copies its own tiles, NS of them ahead: a slot's
    // next K is requested once its K has been read, its next V once its V has.
    auto slotK = [&](uint32_t i) { return smem + (warp * NS + i % NS) * 2 * L::kTileBytes; };
    auto scaleK = [&](uint32_t i) { return reinterpret_cast<float *>(smem + L::kScales) + (warp * NS + i % NS) * 2 * T; };
    const uint32_t stride = p.nKV * HD;
    const uint8_t *storeK = reinterpret_cast<const uint8_t *>(p.k8w) + static_cast<size_t>(kvHead) * HD;
    const uint8_t *storeV = reinterpret_cast<const uint8_t *>(p.v8w) + static_cast<size_t>(kvHead) * HD;
    // the warp that takes the last tile stores the token's row; into the tile itself when that is among its first ones
    const bool append = !ROWS && p.appendK != nullptr && t1 == len && nTiles != 0;
    const uint64_t newRow = rowBase + (!ROWS && p.devLens ? p.devLens[b] + p.lenAdd : len) - 1u;
    // a device length outside the pool (or no length at all): no row written
    const bool outside = (append && newRow >= p.totalRows) || (!ROWS && p.appendK != nullptr && len == 0u);
    if (outside && lane == 0) atomicOr(p.err, kDevErrRowBound);
    const bool mine = append && !outside && (nTiles - 1u) % SW == sw;
    const bool intoTile = mine && (nTiles - 1u) / SW < NS;
    const uint64_t have = intoTile ? rowBase + len - 1u : min(rowBase + len, p.totalRows);
    auto request = [&](uint32_t i, bool isV) {
        const uint32_t j = sw + i * SW;
        if (j < nTiles) {
            const uint64_t row = rowBase + t0 + j * T;
            const uint32_t count = have > row ? static_cast<uint32_t>(min(have - row, static_cast<uint64_t>(T))) : 0u;
            copyTile<T, HD>(smemAddr(slotK(i) + (isV ? L::kTileBytes : 0)), isV ? storeV : storeK, stride, row, count, lane);
            if (lane < count) cpAsync4(scaleK(i) + (isV ? T : 0) + lane, (isV ? p.vs : p.ks) + (row + lane) * p.nKV + kvHead);
        }
        cpAsyncCommit();
    };
    auto requestK = [&](uint32_t i) { request(i, false); };
    auto requestV = [&](uint32_t i) { request(i, true); };
    NewQuantRow<HD, T> fresh;
    const size_t newSrc = (static_cast<size_t>(b) * p.nKV + kvHead) * HD;
    // (behind the loads of q: queued behind 128 KB of tiles of the SM, q came 3.7 us after the dependency:
    // 16 / 2 / 256, norm and gate included, 16383 rows 16.1 -> 15.1 us a layer, 8 / 4 / 256 at 8000 rows 14.8 -> 13.5.  Causal rows, tiles
    // first -> this: 28 / 4 / 128, 64 rows 7.6 -> 6.55 us, 512 behind 2000 199 -> 188; 16 / 2 / 256, 64 rows 6.15 -> 4.9, 512 behind 2000
    // 199 -> 194.  There the loop is not unrolled and q goes through the read-only path: without that, 2 rows behind 16000
    // took 91.4 and 177.6 us, with the tiles first 90.8 and 176.2, like this 88.4 and 175.5.)
    auto requestFirst = [&]() {
        if (mine) fresh.load(p.appendK + newSrc, p.appendV + newSrc, lane);
#pragma unroll(ROWS ? 1 : NS)
        for (uint32_t i = 0; i < NS; ++i) {
            requestK(i);
            requestV(i);
        }
    };

    const uint32_t g = lane >> 2, t = lane & 3u;
    // What MMA column j (0..7) of this warp stands for.
    auto colValid = [&](uint32_t j) { return ROWS ? (b * 8u + j < p.qRows) : (p.colBase + j < p.group); };
    auto colIndex = [&](uint32_t j) -> size_t {  // index of the column's q / out vector, in units of HD
        return ROWS ? (static_cast<size_t>(b) * 8u + j) * p.nHeads + hg
                    : static_cast<size_t>(b) * p.nHeads + kvHead * p.group + p.colBase + j;
    };
    // exclusive row bound of a column: everything in decode, causal in rows mode
    auto colLen = [&](uint32_t j) { return ROWS ? min(t1, rowsPos + b * 8u + j + 1u) : t1; };

    I8Query<HD> qf;
    const float *qp = p.q + colIndex(colValid(g) ? g : 0) * HD;
    if constexpr (ROWS) i8LoadQuery<HD>(qf, qp, colValid(g), p.invSqrt, lane, requestFirst);
    else i8LoadQueryShared<HD, NW, 0>(qf, smem + L::kQuery, qp, colValid(g), p.invSqrt, warp, lane, requestFirst);
    if (mine) {
        const size_t dst = newRow * p.nKV + kvHead;
        const uint32_t i = (nTiles - 1u) / SW;
        float4 *mk = nullptr, *mv = nullptr;
        if (p.mir.k != nullptr)
            mk = reinterpret_cast<float4 *>(p.mir.k) + dst * (HD / 4), mv = reinterpret_cast<float4 *>(p.mir.v) + dst * (HD / 4);
        uint8_t *tile = intoTile ? slotK(i) : nullptr;
        fresh.store(p.k8w + dst * (HD / 4), p.v8w + dst * (HD / 4), const_cast<float *>(p.ks) + dst, const_cast<float *>(p.vs) + dst,
                    mk, mv, tile, tile + L::kTileBytes, scaleK(i), scaleK(i) + T, len - 1u - (t0 + (nTiles - 1u) * T), lane);
        __syncwarp();
    }
    const uint32_t len0 = colLen(2 * t), len1 = colLen(2 * t + 1);

    float m0 = kNegBig, m1 = kNegBig, l0 = 0.0f, l1 = 0.0f;
    float ps0 = 0.0f, ps1 = 0.0f;  // sum of p*sv as fed to the PV MMA (V bytes enter as x + 128)
    uint32_t Ebits = 0;            // running power-of-two scale of the V row scales (0 = unset)
    float invE = 0.0f;
    float o[NC][4];
#pragma unroll
    for (int i = 0; i < NC; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;

    const uint32_t lr = (lane & 7u) + ((lane >> 3) & 1u) * 8u;  // ldmatrix row this lane addresses
    const uint32_t lco = lane >> 4;                             // and which chunk of the pair
    const uint32_t lmOff = lr * 128;

    for (uint32_t i = 0, tile = sw; tile < nTiles; ++i, tile += SW) {
        cpAsyncWait<2 * NS - 1>();  // K of this tile is in, what was requested behind it may still be on its way
        const float *sK = scaleK(i), *sV = sK + T;
        const uint32_t tokBase = t0 + tile * T + g;
        float svr[NR], sc[NR][2];
        i8Scores<HD, MT>(qf, smemAddr(slotK(i)), sK, tokBase, len0, len1, lane, sc);
        float mx0 = fmaxf(sc[0][0], sc[1][0]), mx1 = fmaxf(sc[0][1], sc[1][1]);
        __syncwarp();  // every lane has read its part of K
        requestK(i + NS);
        cpAsyncWait<2 * NS - 1>();  // V of this tile is in
#pragma unroll
        for (int r = 0; r < NR; ++r) svr[r] = tokBase + 8 * r < t1 ? sV[g + 8 * r] : 0.0f;
        float svmax = fmaxf(svr[0], svr[1]);
#pragma unroll
        for (int r = 2; r < NR; ++r) {
            mx0 = fmaxf(mx0, sc[r][0]);
            mx1 = fmaxf(mx1, sc[r][1]);
            svmax = fmaxf(svmax, svr[r]);
        }
#pragma unroll
        for (int off = 4; off <= 16; off <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
        }
        // lazy reference point: move it only when the maximum ran ahead by 2^8
        const float mn0 = mx0 > m0 + kLazyLog2 ? mx0 : m0;
        const float mn1 = mx1 > m1 + kLazyLog2 ? mx1 : m1;
        // running power-of-two bound of the V scales (keeps p*sv inside fp16)
        uint32_t eb = __reduce_max_sync(0xffffffffu, __float_as_uint(svmax)) & 0x7f800000u;
        eb = min(eb, 253u << 23);
        float fE = 1.0f;
        if (eb > Ebits) {
            const float newInv = __uint_as_float((254u << 23) - eb);
            fE = Ebits ? __uint_as_float(Ebits) * newInv : 1.0f;
            Ebits = eb;
            invE = newInv;
        }
        if (__any_sync(0xffffffffu, mn0 != m0 || mn1 != m1 || fE != 1.0f)) {
            const float a0s = fastExp2(m0 - mn0), a1s = fastExp2(m1 - mn1);
            const float al0 = a0s * fE, al1 = a1s * fE;
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                o[i][0] *= al0;
                o[i][1] *= al1;
                o[i][2] *= al0;
                o[i][3] *= al1;
            }
            l0 *= a0s;
            l1 *= a1s;
            ps0 *= al0;
            ps1 *= al1;
            m0 = mn0;
            m1 = mn1;
        }
        // p, then p * sv scaled into fp16 range, hi + lo, transposed to the B layout
        uint32_t bh[MT][2], bl[MT][2];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int r = 2 * mt + hf;
                const float p0 = fastExp2(sc[r][0] - m0), p1 = fastExp2(sc[r][1] - m1);
                l0 += p0;
                l1 += p1;
                const float w = svr[r] * invE;
                const float x0 = p0 * w, x1 = p1 * w;
                const uint32_t hi = packHalf2(x0, x1);
                const __half2 hh = *reinterpret_cast<const __half2 *>(&hi);
                const float r0 = x0 - __low2float(hh), r1 = x1 - __high2float(hh);
                const uint32_t lo = packHalf2(r0, r1);
                const __half2 ll = *reinterpret_cast<const __half2 *>(&lo);
                ps0 += __low2float(hh) + __low2float(ll);
                ps1 += __high2float(hh) + __high2float(ll);
                bh[mt][hf] = movmatrixTrans(hi);
                bl[mt][hf] = movmatrixTrans(lo);
            }
        }
        // ---- O^T += V^T . P^T (HD dims x 8 heads), V bytes read transposed ----
        const uint32_t vTile = smemAddr(slotK(i) + L::kTileBytes);
#pragma unroll
        for (int cp = 0; cp < NC / 2; ++cp) {
            const uint32_t at = (((2 * (cp & 3) + lco) ^ (lr & 7u)) << 4) + (cp >> 2) * L::kHalfBytes;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                uint32_t r0, r1, r2, r3;
                ldmatrixX4Trans(r0, r1, r2, r3, vTile + mt * 2048 + lmOff + at);
                r0 ^= 0x80808080u;
                r1 ^= 0x80808080u;
                r2 ^= 0x80808080u;
                r3 ^= 0x80808080u;
                {
                    // rows g / g+8 of this MMA tile are dims 16c+2g / 16c+2g+1, c = 2cp
                    const uint32_t a0 = subnormalPair<0x4240>(r0), a1 = subnormalPair<0x4341>(r0),
                                   a2 = subnormalPair<0x4240>(r1), a3 = subnormalPair<0x4341>(r1);
                    mmaF16(o[2 * cp], a0, a1, a2, a3, bh[mt][0], bh[mt][1]);
                    mmaF16(o[2 * cp], a0, a1, a2, a3, bl[mt][0], bl[mt][1]);
                }
                {
                    const uint32_t a0 = subnormalPair<0x4240>(r2), a1 = subnormalPair<0x4341>(r2),
                                   a2 = subnormalPair<0x4240>(r3), a3 = subnormalPair<0x4341>(r3);
                    mmaF16(o[2 * cp + 1], a0, a1, a2, a3, bh[mt][0], bh[mt][1]);
                    mmaF16(o[2 * cp + 1], a0, a1, a2, a3, bl[mt][0], bl[mt][1]);
                }
            }
        }
        __syncwarp();
        requestV(i + NS);
    }

    // ---- fold the consumer warps of each kv head, write the chunk partial ----
#pragma unroll
    for (int off = 4; off <= 16; off <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, off);
        l1 += __shfl_xor_sync(0xffffffffu, l1, off);
        ps0 += __shfl_xor_sync(0xffffffffu, ps0, off);
        ps1 += __shfl_xor_sync(0xffffffffu, ps1, off);
    }
    namedBarSync(1, NW * 32);  // every consumer is done reading the ring
    float *scr = reinterpret_cast<float *>(smem);
    using F = FoldScratch<HD>;
    constexpr int kWarpScr = F::kWarp;
    float *wO = scr + warp * kWarpScr;  // [8 heads][FoldScratch::kRow], then m[8], l[8]
    {
        // true accumulator = 2^24 * raw - 128 * sum(p*sv), then back from the E-scaled domain
        const float E = __uint_as_float(Ebits);
        const float c0 = 128.0f * ps0, c1 = 128.0f * ps1;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = 16 * c + 2 * g;
            *reinterpret_cast<float2 *>(wO + (2 * t) * F::kRow + d) =
                    make_float2(fmaf(o[c][0], k2p24, -c0) * E, fmaf(o[c][2], k2p24, -c0) * E);
            *reinterpret_cast<float2 *>(wO + (2 * t + 1) * F::kRow + d) =
                    make_float2(fmaf(o[c][1], k2p24, -c1) * E, fmaf(o[c][3], k2p24, -c1) * E);
        }
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
        f.numChunks = p.numChunks, f.slot = blockIdx.x / clusterSize();
        f.firstHead = static_cast<uint32_t>(colIndex(0)), f.nValid = min(8u, p.group - p.colBase);
        f.direct = p.directOut;
        f.qRot = nullptr, f.cosT = nullptr, f.sinT = nullptr, f.tableRow = 0;
        clusterFold<HD, NW>(scr, f, threadIdx.x);
        return;
    }
    constexpr uint32_t V4 = HD / 4;
    for (uint32_t idx = threadIdx.x; idx < 8 * V4; idx += NW * 32) {
        const uint32_t d4 = idx % V4, j = idx / V4;
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

// The split at head_dim 256.  Which tokens one warp accumulates in a row decides the roundings of the result: the V
// bytes enter the products with an offset of 128 that is taken out at the end, so the running sums are large next to the
// result.  Short runs keep that small, and the runs stay what they are whatever the blocks look like: chunks of
// planDecode (one wave of blocks that stream up to four kv heads), a chunk's tokens dealt to 8 / hpc warps.  A block of eight
// warps takes as many neighbouring chunks as fill it: it prepares the query once, and leaves one partial.
// (16 / 2 heads, norm, decode and gate of a layer: a block per chunk with one slot per warp -> this: 2000 rows 12.05 -> 10.05 us, now
// one cluster, 16383 rows 17.1 -> 16.05; 16 / 4: 2000 rows 12.6 -> 9.9, 60000 rows 35.2 -> 31.6; 20 rows of 16 / 2 9.48 -> 9.6.)
static ClusterPlan decodeI8Plan(const tc_decode_i8_batch *d, uint32_t chunksPerBlock, const uint32_t *maxClusters) {
    const DecodePlan dp = planDecode(d->batch, d->nKV, d->maxLen, d->numChunks, 8u * 16u, d->lens == nullptr);
    const uint32_t blocks = (dp.chunksPerSeq + chunksPerBlock - 1u) / chunksPerBlock;
    ClusterPlan best = {1, blocks, dp.chunkTokens};
    // up to 16 blocks one cluster per kv head folds them all; more take the merge
    for (uint32_t lg = 1; lg < 5; ++lg)
        if (blocks > 1 && blocks <= (1u << lg) && maxClusters[lg] >= d->nKV * d->batch) {
            best.cluster = 1u << lg, best.clusters = 1;
            break;
        }
    return best;
}

template <int SW>
static int decodeI8Hd256(const tc_decode_i8_batch *d, DecodeI8Params prm, cudaStream_t st) {
    constexpr int HD = 256, NW = 8, NS = 2;
    using L = DecodeI8Smem<HD, NW, NS, 1, false>;
    auto kern = decodeI8Kernel<HD, NW, SW, NS, 1, false>;
    static ClusterSetup setup;
    const uint32_t *limits = nullptr;
    int rc = setupCluster(setup, kern, NW * 32, L::kTotal, &limits);
    if (rc != TC_OK) return rc;
    const ClusterPlan pl = decodeI8Plan(d, NW / SW, limits);
    const bool direct = pl.clusters == 1 && !d->partialsOnly;
    if (!direct)
        TC_REQUIRE(d->pAcc && d->pM && d->pL, TC_EWORKSPACE, "decode_i8: partial buffers are required");
    if (d->chunksUsed) *d->chunksUsed = pl.clusters;
    prm.chunkTokens = pl.chunkTokens;
    prm.directOut = direct ? 1 : 0;
    // a launch serves 8 q heads per kv head (the MMA columns); wider groups take one launch per
    // block of 8 and stream the rows again
    for (uint32_t cb = 0; cb < prm.group; cb += 8) {
        prm.colBase = cb;
        if (cb) prm.appendK = prm.appendV = nullptr;  // the row is in
        rc = launchDependent(kern, dim3(pl.clusters * pl.cluster, d->nKV, d->batch), NW * 32, L::kTotal, st, pl.cluster,
                             prm);
        if (rc != TC_OK) return rc;
    }
    if (direct || d->partialsOnly) return TC_OK;
    // merge: the active partial count of a sequence follows from its length (read on
    // the device when the length lives there); slots past it were never written.
    return launchMerge(d->pAcc, d->pM, d->pL, d->out, d->batch, d->nHeads, d->numChunks, pl.clusters, HD, d->lens, prm.lenAdd,
                       pl.chunkTokens * (NW / SW) * pl.cluster, nullptr, true, st);
}

static int i8Params(const tc_decode_i8_batch *d, uint32_t lenHost, uint32_t lenAdd, const F32Mirror &mir, DecodeI8Params *o) {
    memset(o, 0, sizeof(*o));
    o->q = d->q;
    o->out = d->out;
    o->ks = d->ks;
    o->vs = d->vs;
    o->pAcc = d->pAcc;
    o->pM = d->pM;
    o->pL = d->pL;
    o->devLens = d->lens;
    o->devRowBase = d->rowBase;
    o->rowsPerSeq = d->rowsPerSeq;
    o->totalRows = d->totalRows;
    o->lenHost = lenHost;
    o->lenAdd = lenAdd;
    o->nHeads = d->nHeads;
    o->nKV = d->nKV;
    o->group = d->nHeads / d->nKV;
    o->numChunks = d->numChunks;
    o->appendK = d->appendK;
    o->appendV = d->appendV;
    o->k8w = reinterpret_cast<uint32_t *>(const_cast<int8_t *>(d->k8));
    o->v8w = reinterpret_cast<uint32_t *>(const_cast<int8_t *>(d->v8));
    o->mir = mir;
    o->invSqrt = d->invSqrt;
    o->err = devErrorWord();
    TC_REQUIRE(o->err != nullptr, TC_ECUDA, "decode_i8: no device error word");
    return TC_OK;
}

int decodeI8Streams(const tc_decode_i8_batch *d, uint32_t lenHost, uint32_t lenAdd, cudaStream_t st) {
    TC_REQUIRE(d->hd == 128 || d->hd == 256, TC_EUNSUPPORTED, "decode_i8: head_dim %u (built for 128 and 256)", d->hd);
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(d->k8) | reinterpret_cast<uintptr_t>(d->v8) |
                 reinterpret_cast<uintptr_t>(d->q) | reinterpret_cast<uintptr_t>(d->out) |
                 reinterpret_cast<uintptr_t>(d->appendK) | reinterpret_cast<uintptr_t>(d->appendV)) & 15u) == 0,
               TC_EINVAL, "decode_i8: q/out/k8/v8 and the new row need 16-byte alignment");
    DecodeI8Params prm;
    const int rc = i8Params(d, lenHost, lenAdd, F32Mirror{nullptr, nullptr}, &prm);
    if (rc != TC_OK) return rc;
    prm.directOut = 1;
    return launchStreamsI8(prm, d->hd, st);
}

int decodeI8Common(const tc_decode_i8_batch *d, uint32_t lenHost, uint32_t lenAdd, const F32Mirror &mir, cudaStream_t st) {
    TC_REQUIRE(d->q && d->out && d->k8 && d->v8 && d->ks && d->vs, TC_EINVAL, "decode_i8: null pointer");
    TC_REQUIRE(d->hd == 128 || d->hd == 256, TC_EUNSUPPORTED, "decode_i8: head_dim %u (built for 128 and 256)",
               d->hd);
    TC_REQUIRE(d->nKV > 0 && d->nHeads % d->nKV == 0, TC_EINVAL, "decode_i8: nHeads %u not a multiple of nKV %u",
               d->nHeads, d->nKV);
    const uint32_t group = d->nHeads / d->nKV;
    TC_REQUIRE(group <= 64, TC_EUNSUPPORTED, "decode_i8: %u q heads per kv head (built for <= 64)", group);
    TC_REQUIRE(d->batch >= 1 && d->batch <= 65535, TC_EINVAL, "decode_i8: batch %u", d->batch);
    TC_REQUIRE(d->maxLen >= 1, TC_EINVAL, "decode_i8: empty context");
    TC_REQUIRE(d->totalRows >= 1 && d->totalRows < (1ull << 31), TC_EUNSUPPORTED,
               "decode_i8: pool of %llu rows", (unsigned long long) d->totalRows);
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(d->k8) | reinterpret_cast<uintptr_t>(d->v8) |
                 reinterpret_cast<uintptr_t>(d->q) | reinterpret_cast<uintptr_t>(d->out)) & 15u) == 0,
               TC_EINVAL, "decode_i8: q/out/k8/v8 need 16-byte alignment");
    TC_REQUIRE(d->numChunks >= 1, TC_EWORKSPACE, "decode_i8: no chunk slots");
    TC_REQUIRE((d->appendK == nullptr) == (d->appendV == nullptr), TC_EINVAL, "decode_i8: appendK and appendV come together");
    // (the launch moves the new row, and its f32 copy, 16 bytes at a time)
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(d->appendK) | reinterpret_cast<uintptr_t>(d->appendV) |
                 reinterpret_cast<uintptr_t>(mir.k) | reinterpret_cast<uintptr_t>(mir.v)) & 15u) == 0,
               TC_EINVAL, "decode_i8: the new row needs 16-byte alignment");
    // head_dim 128 runs on the tcgen05 integer path
    if (d->hd == 128) return decodeI8Tc(d, lenHost, lenAdd, mir, st);

    // a new row that the host can tell to lie outside the pool (the quantise launch's check; head_dim 128 leaves it to the device)
    const uint64_t lastRow = static_cast<uint64_t>(d->batch - 1) * d->rowsPerSeq + lenHost - 1;
    TC_REQUIRE(d->appendK == nullptr || d->lens != nullptr || d->rowBase != nullptr || lastRow < d->totalRows, TC_ECONTEXT_FULL,
               "decode_i8: row %u of sequence %u passes the pool's %llu rows", lenHost - 1, d->batch - 1,
               (unsigned long long) d->totalRows);
    DecodeI8Params prm;
    const int rc = i8Params(d, lenHost, lenAdd, mir, &prm);
    if (rc != TC_OK) return rc;
    // warps that share a chunk's tokens, by the kv heads (see decodeI8Plan)
    if (d->nKV % 4u == 0) return decodeI8Hd256<2>(d, prm, st);
    if (d->nKV % 2u == 0) return decodeI8Hd256<4>(d, prm, st);
    return decodeI8Hd256<8>(d, prm, st);
}

template <int HD, int MT>
static int launchRowsI8(const DecodeI8Params &prm, cudaStream_t st) {
    constexpr int NW = 8, NS = 3;
    using L = DecodeI8Smem<HD, NW, NS, MT, true>;
    auto kern = decodeI8Kernel<HD, NW, NW, NS, MT, true>;
    static bool attrDone[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attrDone[dev]) {
        TC_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal));
        attrDone[dev] = true;
    }
    return launchDependent(kern, dim3(1, prm.nHeads, (prm.qRows + 7) / 8), NW * 32, L::kTotal, st, 1, prm);
}

// Causal prefill over the int8 store: the decode kernel with query rows as MMA columns.
static int prefillI8(const float *q, const int8_t *k8, const int8_t *v8, const float *ks, const float *vs,
                     float *out, uint32_t seqLen, uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t cachePos,
                     const uint32_t *devPos, uint64_t totalRows, float invSqrt, cudaStream_t st) {
    TC_REQUIRE(q && k8 && v8 && ks && vs && out, TC_EINVAL, "prefill_i8: null pointer");
    TC_REQUIRE(hd == 128 || hd == 256, TC_EUNSUPPORTED, "prefill_i8: head_dim %u (built for 128 and 256)", hd);
    TC_REQUIRE(nKV > 0 && nHeads % nKV == 0, TC_EINVAL, "prefill_i8: nHeads %u not a multiple of nKV %u", nHeads,
               nKV);
    TC_REQUIRE(totalRows >= 1 && totalRows < (1ull << 31), TC_EUNSUPPORTED, "prefill_i8: pool of %llu rows",
               (unsigned long long) totalRows);
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(k8) | reinterpret_cast<uintptr_t>(v8) | reinterpret_cast<uintptr_t>(q) |
                 reinterpret_cast<uintptr_t>(out)) & 15u) == 0,
               TC_EINVAL, "prefill_i8: q/out/k8/v8 need 16-byte alignment");
    if (seqLen == 0) return TC_OK;
    if (devPos == nullptr && static_cast<uint64_t>(cachePos) + seqLen > totalRows) {
        setError("prefill_i8: rows [%u, %llu) pass the pool of %llu rows", cachePos,
                 (unsigned long long) cachePos + seqLen, (unsigned long long) totalRows);
        return TC_ECONTEXT_FULL;
    }
    const uint32_t rowBlocks = (seqLen + 7) / 8;
    TC_REQUIRE(rowBlocks <= 65535 && nHeads <= 65535, TC_EUNSUPPORTED, "prefill_i8: %u rows x %u heads", seqLen,
               nHeads);
    DecodeI8Params prm;
    memset(&prm, 0, sizeof(prm));
    prm.q = q;
    prm.out = out;
    prm.ks = ks;
    prm.vs = vs;
    prm.k8w = reinterpret_cast<uint32_t *>(const_cast<int8_t *>(k8));
    prm.v8w = reinterpret_cast<uint32_t *>(const_cast<int8_t *>(v8));
    prm.totalRows = totalRows;
    prm.nHeads = nHeads;
    prm.nKV = nKV;
    prm.group = nHeads / nKV;
    prm.numChunks = 1;
    prm.qRows = seqLen;
    prm.cachePos = cachePos;
    prm.devPos = devPos;
    prm.invSqrt = invSqrt;
    prm.directOut = 1;
    prm.err = devErrorWord();
    TC_REQUIRE(prm.err != nullptr, TC_ECUDA, "prefill_i8: no device error word");
    if (hd == 256) return launchRowsI8<256, 1>(prm, st);
    return launchRowsI8<128, 2>(prm, st);
}

}  // namespace tc

extern "C" {

int tc_attn_prefill_i8(const float *q, const int8_t *k8, const int8_t *v8, const float *ks, const float *vs,
                       float *out, uint32_t seqLen, uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t cachePos,
                       const uint32_t *devPos, uint64_t totalRows, float invSqrt, tc_stream stream) {
    return tc::prefillI8(q, k8, v8, ks, vs, out, seqLen, nHeads, nKV, hd, cachePos, devPos, totalRows, invSqrt,
                         static_cast<cudaStream_t>(stream));
}

int tc_attn_decode_i8_batch(const tc_decode_i8_batch *d, tc_stream stream) {
    TC_REQUIRE(d != nullptr, TC_EINVAL, "tc_attn_decode_i8_batch: null descriptor");
    return tc::decodeI8Common(d, d->maxLen, 0, tc::F32Mirror{nullptr, nullptr}, static_cast<cudaStream_t>(stream));
}

int tc_attn_decode_i8(const float *q, const int8_t *k8, const int8_t *v8, const float *ks, const float *vs,
                      float *out, float *pAcc, float *pM, float *pL, uint32_t nHeads, uint32_t nKV, uint32_t hd,
                      uint32_t cachePos, const uint32_t *devPos, uint64_t totalRows, uint32_t numChunks,
                      uint32_t chunkSize, float invSqrt, tc_stream stream) {
    (void) chunkSize;
    TC_REQUIRE(static_cast<uint64_t>(cachePos) + 1 <= totalRows, TC_ECONTEXT_FULL,
               "tc_attn_decode_i8: position %u is outside the pool of %llu rows", cachePos,
               (unsigned long long) totalRows);
    tc_decode_i8_batch d;
    memset(&d, 0, sizeof(d));
    d.q = q;
    d.out = out;
    d.k8 = k8;
    d.v8 = v8;
    d.ks = ks;
    d.vs = vs;
    d.pAcc = pAcc;
    d.pM = pM;
    d.pL = pL;
    d.lens = devPos;
    d.rowBase = nullptr;
    d.rowsPerSeq = 0;
    d.totalRows = totalRows;
    d.batch = 1;
    d.nHeads = nHeads;
    d.nKV = nKV;
    d.hd = hd;
    d.maxLen = cachePos + 1;
    d.numChunks = numChunks;
    d.invSqrt = invSqrt;
    return tc::decodeI8Common(&d, cachePos + 1, devPos ? 1u : 0u, tc::F32Mirror{nullptr, nullptr}, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------
// A decode entry point that allocates nothing
// ---------------------------------------------------------------------------------
// Some callers hold no allocator they may use at the moment attention runs: a host
// that hands this library bare device pointers from a memory plan frozen at load
// time, or a latency-critical serving loop that must not touch the device allocator
// once it is running.  For them the split-KV partials (the only scratch this kernel needs)
// live in a fixed array inside the library's own device image instead of in
// caller-provided buffers.  Every GPU that loads the library carries the array
// (kNoAllocBytes, about 5.3 MB) until the process exits.
constexpr uint32_t kNoAllocMaxHeads = 64;    // q heads
constexpr uint32_t kNoAllocChunks = 160;     // chunk slots per head (one per SM and a few spare)
constexpr size_t kNoAllocAccFloats = static_cast<size_t>(kNoAllocMaxHeads) * kNoAllocChunks * tc::kHD;
constexpr size_t kNoAllocMLFloats = static_cast<size_t>(kNoAllocMaxHeads) * kNoAllocChunks;
constexpr size_t kNoAllocBytes = (kNoAllocAccFloats + 2 * kNoAllocMLFloats) * sizeof(float);
static __device__ __align__(256) float g_noAllocScratch[kNoAllocAccFloats + 2 * kNoAllocMLFloats];

// In host code the array's name is only a handle for the runtime, not a device
// address, so the address is asked for once per device (with that device current)
// and remembered.
static int noAllocScratch(float **ptr) {
    static std::mutex mu;
    static float *addr[64] = {nullptr};
    int dev = 0;
    TC_CUDA_OK(cudaGetDevice(&dev));
    TC_REQUIRE(dev >= 0 && dev < 64, TC_EUNSUPPORTED, "tc_attn_decode_i8_noalloc: device ordinal %d", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (addr[dev] == nullptr) {
        void *p = nullptr;
        TC_CUDA_OK(cudaGetSymbolAddress(&p, g_noAllocScratch));
        addr[dev] = static_cast<float *>(p);
    }
    *ptr = addr[dev];
    return TC_OK;
}

int tc_attn_decode_i8_noalloc(const float *q, const int8_t *k8, const int8_t *v8, const float *ks, const float *vs,
                              float *out, uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t cachePos,
                              uint64_t totalRows, float invSqrt, tc_stream stream) {
    TC_REQUIRE(nHeads >= 1 && nHeads <= kNoAllocMaxHeads, TC_EWORKSPACE,
               "tc_attn_decode_i8_noalloc: %u q heads, the built-in scratch holds at most %u", nHeads,
               kNoAllocMaxHeads);
    TC_REQUIRE(hd == static_cast<uint32_t>(tc::kHD), TC_EWORKSPACE,
               "tc_attn_decode_i8_noalloc: head_dim %u, the built-in scratch is laid out for %d", hd, tc::kHD);
    TC_REQUIRE(static_cast<uint64_t>(cachePos) + 1 <= totalRows, TC_ECONTEXT_FULL,
               "tc_attn_decode_i8_noalloc: position %u is outside the pool of %llu rows", cachePos,
               (unsigned long long) totalRows);
    float *scratch = nullptr;
    const int rc = noAllocScratch(&scratch);
    if (rc != TC_OK) return rc;
    tc_decode_i8_batch d;
    memset(&d, 0, sizeof(d));
    d.q = q;
    d.out = out;
    d.k8 = k8;
    d.v8 = v8;
    d.ks = ks;
    d.vs = vs;
    // the three partial arrays are carved out of the one array; nothing in them has to
    // start at zero (the merge reads only the chunk slots this call wrote)
    d.pAcc = scratch;
    d.pM = scratch + kNoAllocAccFloats;
    d.pL = scratch + kNoAllocAccFloats + kNoAllocMLFloats;
    d.totalRows = totalRows;
    d.batch = 1;
    d.nHeads = nHeads;
    d.nKV = nKV;
    d.hd = hd;
    d.maxLen = cachePos + 1;
    d.numChunks = kNoAllocChunks;
    d.invSqrt = invSqrt;
    return tc::decodeI8Common(&d, cachePos + 1, 0u, tc::F32Mirror{nullptr, nullptr}, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
