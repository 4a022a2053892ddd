// decode_i8_streams.cu -- one query token over the int8 store, any length up to the launch's bound, no partial buffers:
// what a captured decode step of the int8 store replays.
//
// What it replaces: kQ35WarpAttention8Prefill / kQ35PrefillAttnSharedKV8 with one query row (include/gpu/
// GpuQwen35Kernels.hpp:2306-2435), the reference's graph-safe form of the int8 decode.
//
// The roundings of the result are those of the causal kernel (decode_i8.cu): its V bytes enter the products with an offset
// of 128 that is taken out at the end, so the running sums are large next to the result and the order in which tiles are
// accumulated shows.  That order is eight streams -- tile j (16 MT tokens) belongs to stream j % 8, a stream's tiles are
// folded one after the other -- and it is kept: a block is a stream, an 8-block cluster a kv head.  Inside a stream only
// three things depend on the tile before: the reference point of the maximum, the scale of the V factors, and the
// accumulators, each dimension on its own.  So
//   * eight score warps take tiles in turn: scores (K product), then -- once the warps of a round have told each other
//     their tiles' maxima and each has walked through them in tile order -- probabilities as MMA operands;
//   * four value warps own HD / 4 dimensions each and walk through all tiles of the stream: rescale, four to eight products;
//   * a sum warp walks along with the row sums.
// A tile costs the walk some 200 cycles where one warp doing all of it took 2500: 5000 rows of 28 q / 4 kv heads of 128
// (157 tiles of 32 tokens, 20 per stream) took 13.8 us, 26 with a warp per stream, 27.5 with a block per q head.
// The walks of values and sums hear of a round of eight tiles at a time, and a round's V tiles are requested when its
// probabilities are out: the score warps used to stand until the walk was through with the round before, and a wait per
// tile cost the walk 170 cycles.  Most tiles move no reference point, and are passed over together.  Per layer, 28 / 4 / 128 at 5000 /
// 8000 / 16000 rows 11.3 / 16.5 / 29.6 -> 10.8 / 14.2 / 23.0 us, 16 / 2 / 256 at 8000 (norm and gate included) 34.4 -> 25.9.
#include "decode_i8.cuh"

namespace tc {

template <int HD, int MT>
struct I8StreamSmem {
    static constexpr int T = 16 * MT, NR = 2 * MT;
    static constexpr int kScoreWarps = 8, kValueWarps = 4, kWarps = kScoreWarps + kValueWarps + 1;
    static constexpr int kSlots = 2 * kScoreWarps;                 // V tiles and probability records in flight
    static constexpr int kHalfBytes = T * 128;                     // half-tile of 128 dims
    static constexpr int kTileBytes = T * HD;
    static constexpr int kRecord = 1536 * MT + 128;                // P operands, P and P x scale per row, factors
    static constexpr int kK = 0;                                   // [score warp][2] K tiles
    static constexpr int kV = kK + kScoreWarps * 2 * kTileBytes;   // [slot] V tiles
    static constexpr int kRec = kV + kSlots * kTileBytes;          // [slot]
    static constexpr int kScales = kRec + kSlots * kRecord;        // [score warp][2][K, V][T]
    static constexpr int kMax = kScales + kScoreWarps * 4 * T * 4; // [2][score warp][12]: column maxima, V scale bits
    static constexpr int kEnd = kMax + 2 * kScoreWarps * 12 * 4;   // m[8], E, then l[8], sums of P x scale [8]
    static constexpr int kBars = kEnd + 32 * 4;                    // full, empty of the even / odd rounds
    // The score warps prepare the query together where it is long (16 / 2 / 256, norm and gate included: 20 / 500 / 2000 / 5000 rows
    // 10.0 / 10.5 / 14.2 / 25.3 -> 9.75 / 10.0 / 13.85 / 24.9 us a layer; 8 / 2 / 128 at 20 rows 5.65 -> 5.9).
    static constexpr bool kShareQuery = HD > 128;
    static constexpr int kQuery = kBars + 4 * 8;                   // the query operands
    static constexpr int kTotal = kQuery + (kShareQuery ? I8QueryShare<HD, kScoreWarps>::kBytes : 0) + 128;
    static_assert(kQuery % 16 == 0, "16-byte accesses");
    static_assert(FoldScratch<HD>::kWarp * 4 <= kV, "the fold reuses the K tiles");
    static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

template <int HD, int MT>
__global__ void __launch_bounds__(I8StreamSmem<HD, MT>::kWarps * 32, 1)
decodeI8StreamsKernel(const __grid_constant__ DecodeI8Params p) {
    using L = I8StreamSmem<HD, MT>;
    constexpr int T = L::T, NR = L::NR;
    constexpr uint32_t SW = L::kScoreWarps, VW = L::kValueWarps, NSLOT = L::kSlots, kThreads = L::kWarps * 32;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t stream = clusterRank(), kvHead = blockIdx.y;

    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 127) & ~uintptr_t(127));
    uint64_t *fullBar = reinterpret_cast<uint64_t *>(smem + L::kBars), *emptyBar = fullBar + 2;
    float *sEnd = reinterpret_cast<float *>(smem + L::kEnd);
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < 2; ++s) {
            mbarInit(&fullBar[s], SW);
            mbarInit(&emptyBar[s], VW + 1);
        }
        fenceBarrierInit();
    }
    __syncthreads();
    clusterHello();
    {
        const size_t row = static_cast<size_t>(kvHead) * HD;
        prefetchToken<HD>(p.q + (static_cast<size_t>(kvHead) * p.group + p.colBase) * HD, min(8u, p.group - p.colBase),
                          p.appendK != nullptr ? p.appendK + row : nullptr, p.appendV + row, nullptr, nullptr, threadIdx.x);
    }
    gridDepWait();

    const uint32_t want = p.devLens ? p.devLens[0] + p.lenAdd : p.lenHost;
    const uint32_t len = min(want, p.lenHost);  // (the host's length is the upper bound of a device length)
    const uint32_t nTiles = (len + T - 1) / T;
    const uint32_t n = nTiles > stream ? (nTiles - stream + 7u) / 8u : 0u;  // tiles of this stream: stream + 8 i
    // the block that stores the token's row lets the next grid start behind that store: it may request the row early
    // (a device position outside the pool, the one whose length wraps to 0 among them, stores none)
    const bool outside = p.appendK != nullptr && want - 1u >= p.totalRows;
    const bool storesRow = p.appendK != nullptr && !outside && (nTiles - 1u) % 8u == stream;
    if (!storesRow) gridDepLaunch();
    const uint32_t head0 = kvHead * p.group + p.colBase, nValid = min(8u, p.group - p.colBase);
    // record of a slot: P operands [MT][32 lanes] uint4, P [2 NR][32], P x scale [2 NR][32], then al[8], as[8], flag
    auto record = [&](uint32_t i) { return smem + L::kRec + (i % NSLOT) * L::kRecord; };
    constexpr uint32_t kRecP = 512 * MT, kRecX = 1024 * MT, kRecF = 1536 * MT;

    const uint32_t lr = (lane & 7u) + ((lane >> 3) & 1u) * 8u, lco = lane >> 4;  // ldmatrix row and chunk of this lane
    constexpr int CP = HD / 128;  // 32-dim groups of a value warp
    float o[2 * CP][4];           // its accumulators, by 16-dim group
#pragma unroll
    for (int c = 0; c < 2 * CP; ++c) o[c][0] = o[c][1] = o[c][2] = o[c][3] = 0.0f;

    if (warp < SW) {
        // ---------------------------------- scores and probabilities ----------------------------------
        const uint32_t stride = p.nKV * HD;
        const uint8_t *storeK = reinterpret_cast<const uint8_t *>(p.k8w) + static_cast<size_t>(kvHead) * HD;
        const uint8_t *storeV = reinterpret_cast<const uint8_t *>(p.v8w) + static_cast<size_t>(kvHead) * HD;
        auto slotK = [&](uint32_t i) { return smem + L::kK + (warp * 2 + (i / SW) % 2) * L::kTileBytes; };
        auto scales = [&](uint32_t i) { return reinterpret_cast<float *>(smem + L::kScales) + (warp * 2 + (i / SW) % 2) * 2 * T; };
        // the warp that takes the last tile stores the token's row; into the tile itself when it is the warp's first one
        if (outside && stream == 0 && threadIdx.x == 0) atomicOr(p.err, kDevErrRowBound);
        const uint32_t iLast = (nTiles - 1u) / 8u;
        const bool hasRow = storesRow && iLast % SW == warp;
        const bool intoTile = hasRow && iLast < SW;
        const uint32_t have = intoTile ? len - 1u : static_cast<uint32_t>(min(static_cast<uint64_t>(len), p.totalRows));
        auto request = [&](uint32_t i, bool isV) {
            const uint32_t row = (stream + 8u * i) * T;
            uint8_t *tile = isV ? smem + L::kV + (i % NSLOT) * L::kTileBytes : slotK(i);
            const uint32_t count = have > row ? min(have - row, static_cast<uint32_t>(T)) : 0u;
            copyTile<T, HD>(smemAddr(tile), isV ? storeV : storeK, stride, row, count, lane);
            if (lane < count)
                cpAsync4(scales(i) + (isV ? T : 0) + lane, (isV ? p.vs : p.ks) + static_cast<size_t>(row + lane) * p.nKV + kvHead);
        };
        auto requestK = [&](uint32_t i) {
            if (i < n) request(i, false);
            cpAsyncCommit();
        };
        bool ok = true;
        auto requestV = [&](uint32_t i) {
            if (ok && i < n) {
                // the tiles of two rounds before have been folded by everybody
                if (i >= NSLOT) ok = mbarWait(&emptyBar[(i / SW) & 1u], (i / NSLOT - 1u) & 1u, p.err, kDevErrEmptyWait);
                request(i, true);
            }
            cpAsyncCommit();
        };
        NewQuantRow<HD, T> fresh;
        const size_t newSrc = static_cast<size_t>(kvHead) * HD;
        // (behind the loads of q, which would queue behind the tiles' otherwise; the tile after the first one is requested behind
        // the row's store when it holds the row)
        auto requestFirst = [&]() {
            if (hasRow) fresh.load(p.appendK + newSrc, p.appendV + newSrc, lane);
            requestK(warp);
            requestV(warp);
            if (!hasRow) requestK(warp + SW);
        };
        I8Query<HD> qf;
        const float *qp = p.q + static_cast<size_t>(head0 + (g < nValid ? g : 0u)) * HD;
        if constexpr (L::kShareQuery) i8LoadQueryShared<HD, SW, 1>(qf, smem + L::kQuery, qp, g < nValid, p.invSqrt, warp, lane, requestFirst);
        else i8LoadQuery<HD>(qf, qp, g < nValid, p.invSqrt, lane, requestFirst);
        if (hasRow) {
            const size_t dst = static_cast<size_t>(len - 1u) * p.nKV + kvHead;
            uint8_t *tile = intoTile ? slotK(iLast) : nullptr;
            fresh.store(p.k8w + dst * (HD / 4), p.v8w + dst * (HD / 4), const_cast<float *>(p.ks) + dst,
                        const_cast<float *>(p.vs) + dst, nullptr, nullptr, tile, smem + L::kV + (iLast % NSLOT) * L::kTileBytes,
                        scales(iLast), scales(iLast) + T, len - 1u - (nTiles - 1u) * T, lane);
            __syncwarp();
            requestK(warp + SW);
        }
        float *sMax = reinterpret_cast<float *>(smem + L::kMax);
        float m0 = kNegBig, m1 = kNegBig;  // at the start of the round
        uint32_t Ebits = 0;                // running power-of-two scale of the V row scales (0 = unset)
        for (uint32_t round = 0; round * SW < n; ++round) {
            const uint32_t i = round * SW + warp;
            cpAsyncWait<2>();  // K of this tile is in
            const uint32_t tokBase = (stream + 8u * i) * T + g;
            float sc[NR][2], svr[NR];
            float mx0 = -INFINITY, mx1 = -INFINITY, svmax = 0.0f;
            if (i < n) {  // warp-uniform
                i8Scores<HD, MT>(qf, smemAddr(slotK(i)), scales(i), tokBase, len, len, lane, sc);
                __syncwarp();
            }
            requestK(i + 2 * SW);  // (every lane is through with K)
            cpAsyncWait<1>();      // V of this tile is in
            if (i < n) {
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    svr[r] = tokBase + 8 * r < len ? scales(i)[T + g + 8 * r] : 0.0f;
                    mx0 = fmaxf(mx0, sc[r][0]);
                    mx1 = fmaxf(mx1, sc[r][1]);
                    svmax = fmaxf(svmax, svr[r]);
                }
#pragma unroll
                for (int off = 4; off <= 16; off <<= 1) {
                    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
                    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
                }
            }
            const uint32_t ebMine = min(__reduce_max_sync(0xffffffffu, __float_as_uint(svmax)) & 0x7f800000u, 253u << 23);
            // ---- the round's maxima, in tile order ----
            float *mine = sMax + ((round & 1u) * SW + warp) * 12u;
            if (g == 0) *reinterpret_cast<float2 *>(mine + 2 * t) = make_float2(mx0, mx1);
            if (lane == 0) mine[8] = __uint_as_float(ebMine);
            namedBarSync(1, SW * 32);
            float a0 = 1.0f, a1 = 1.0f, fMine = 1.0f, r0 = m0, r1 = m1;
            uint32_t eMine = Ebits;
            bool moved = false;
            float2 mx[SW];
            uint32_t eb[SW];
#pragma unroll
            for (uint32_t w = 0; w < SW; ++w) {
                const float *other = sMax + ((round & 1u) * SW + w) * 12u;
                mx[w] = *reinterpret_cast<const float2 *>(other + 2 * t);
                eb[w] = __float_as_uint(other[8]);
            }
            // Tiles that move nothing for any head -- nearly all behind the first -- are passed over together; the others one
            // after the other.
            uint32_t todo = (1u << SW) - 1u;
            while (true) {
                uint32_t moves = 0;
#pragma unroll
                for (uint32_t w = 0; w < SW; ++w)
                    moves |= mx[w].x > m0 + kLazyLog2 || mx[w].y > m1 + kLazyLog2 || eb[w] > Ebits ? 1u << w : 0u;
                moves = __reduce_or_sync(0xffffffffu, moves) & todo;
                if (moves == 0u) break;
                const uint32_t f = __ffs(moves) - 1u;
                float2 top = mx[0];
                uint32_t e = eb[0];
#pragma unroll
                for (uint32_t w = 1; w < SW; ++w)
                    if (w == f) top = mx[w], e = eb[w];
                // lazy reference point: move it only when the maximum ran ahead by 2^8
                const float mn0 = top.x > m0 + kLazyLog2 ? top.x : m0;
                const float mn1 = top.y > m1 + kLazyLog2 ? top.y : m1;
                float fE = 1.0f;
                if (e > Ebits) {
                    fE = Ebits ? __uint_as_float(Ebits) * __uint_as_float((254u << 23) - e) : 1.0f;
                    Ebits = e;
                }
                if (f == warp) {
                    a0 = fastExp2(m0 - mn0), a1 = fastExp2(m1 - mn1), fMine = fE;
                    moved = mn0 != m0 || mn1 != m1 || fE != 1.0f;
                }
                m0 = mn0, m1 = mn1;
                if (f <= warp) r0 = m0, r1 = m1, eMine = Ebits;
                todo = ~((2u << f) - 1u);
            }
            const float invE = eMine ? __uint_as_float((254u << 23) - eMine) : 0.0f;
            const bool any = __any_sync(0xffffffffu, moved);
            if (i < n) {
                // ---- p, then p * sv scaled into fp16 range, hi + lo, transposed to the B layout ----
                uint8_t *rec = record(i);
                float *recP = reinterpret_cast<float *>(rec + kRecP) + lane, *recX = reinterpret_cast<float *>(rec + kRecX) + lane;
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    uint32_t bh[2], bl[2];
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const int r = 2 * mt + hf;
                        const float p0 = fastExp2(sc[r][0] - r0), p1 = fastExp2(sc[r][1] - r1);
                        const float w = svr[r] * invE;
                        const float x0 = p0 * w, x1 = p1 * w;
                        const uint32_t hi = packHalf2(x0, x1);
                        const __half2 hh = *reinterpret_cast<const __half2 *>(&hi);
                        const float d0 = x0 - __low2float(hh), d1 = x1 - __high2float(hh);
                        const uint32_t lo = packHalf2(d0, d1);
                        const __half2 ll = *reinterpret_cast<const __half2 *>(&lo);
                        recP[(2 * r) * 32] = p0, recP[(2 * r + 1) * 32] = p1;
                        recX[(2 * r) * 32] = __low2float(hh) + __low2float(ll);
                        recX[(2 * r + 1) * 32] = __high2float(hh) + __high2float(ll);
                        bh[hf] = movmatrixTrans(hi);
                        bl[hf] = movmatrixTrans(lo);
                    }
                    *reinterpret_cast<uint4 *>(rec + (mt * 32 + lane) * 16) = make_uint4(bh[0], bh[1], bl[0], bl[1]);
                }
                float *fac = reinterpret_cast<float *>(rec + kRecF);
                if (g == 0) {
                    *reinterpret_cast<float2 *>(fac + 2 * t) = make_float2(a0 * fMine, a1 * fMine);
                    *reinterpret_cast<float2 *>(fac + 8 + 2 * t) = make_float2(a0, a1);
                }
                if (lane == 0) *reinterpret_cast<uint32_t *>(fac + 16) = any ? 1u : 0u;
            }
            __syncwarp();
            // (a warp whose wait ran out stays with the others' barrier and hands nothing on: their waits end too)
            if (ok && lane == 0) mbarArrive(&fullBar[round & 1u]);
            requestV(i + SW);  // (waits for the values of the round before, which are folded under this one)
            if (hasRow && round == 0) {
                // (here the row's stores are long done: right behind them the fence cost 0.5 us of the step)
                __threadfence();
                __syncwarp();
                gridDepLaunch();
            }
        }
        if (warp == 0) {
            if (g == 0) sEnd[2 * t] = m0, sEnd[2 * t + 1] = m1;
            if (lane == 0) sEnd[8] = __uint_as_float(Ebits);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < SW + VW) {
        // ---------------------------------- accumulators ----------------------------------
        const uint32_t cp0 = (warp - SW) * CP;  // dims 32 cp0 .. 32 (cp0 + CP) - 1
        for (uint32_t i0 = 0, round = 0; i0 < n; i0 += SW, ++round) {
            if (!mbarWait(&fullBar[round & 1u], (round >> 1) & 1u, p.err, kDevErrFullWait)) break;
            const uint32_t i1 = min(n, i0 + SW);
#pragma unroll 2
            for (uint32_t i = i0; i < i1; ++i) {
                const uint8_t *rec = record(i);
                const float *fac = reinterpret_cast<const float *>(rec + kRecF);
                uint4 b[MT];
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) b[mt] = *reinterpret_cast<const uint4 *>(rec + (mt * 32 + lane) * 16);
                uint32_t v[CP][MT][4];
                const uint32_t vTile = smemAddr(smem + L::kV + (i % NSLOT) * L::kTileBytes) + lr * 128;
#pragma unroll
                for (int c = 0; c < CP; ++c) {
                    const uint32_t cp = cp0 + c;
                    const uint32_t sw = (((2 * (cp & 3u) + lco) ^ (lr & 7u)) << 4) + (cp >> 2) * L::kHalfBytes;
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
                        ldmatrixX4Trans(v[c][mt][0], v[c][mt][1], v[c][mt][2], v[c][mt][3], vTile + mt * 2048 + sw);
                }
                if (*reinterpret_cast<const uint32_t *>(fac + 16) != 0u) {
                    const float2 al = *reinterpret_cast<const float2 *>(fac + 2 * t);
#pragma unroll
                    for (int c = 0; c < 2 * CP; ++c) o[c][0] *= al.x, o[c][1] *= al.y, o[c][2] *= al.x, o[c][3] *= al.y;
                }
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    // rows g / g + 8 of an MMA tile are dims 16 c + 2 g / 16 c + 2 g + 1
                    uint32_t x[2 * CP][4];
#pragma unroll
                    for (int c = 0; c < 2 * CP; ++c) {
                        const uint32_t r0 = v[c / 2][mt][c % 2 * 2] ^ 0x80808080u, r1 = v[c / 2][mt][c % 2 * 2 + 1] ^ 0x80808080u;
                        x[c][0] = subnormalPair<0x4240>(r0), x[c][1] = subnormalPair<0x4341>(r0);
                        x[c][2] = subnormalPair<0x4240>(r1), x[c][3] = subnormalPair<0x4341>(r1);
                    }
#pragma unroll
                    for (int c = 0; c < 2 * CP; ++c) mmaF16(o[c], x[c][0], x[c][1], x[c][2], x[c][3], b[mt].x, b[mt].y);
#pragma unroll
                    for (int c = 0; c < 2 * CP; ++c) mmaF16(o[c], x[c][0], x[c][1], x[c][2], x[c][3], b[mt].z, b[mt].w);
                }
            }
            __syncwarp();
            if (lane == 0) mbarArrive(&emptyBar[round & 1u]);
        }
    } else {
        // ---------------------------------- row sums ----------------------------------
        float l0 = 0.0f, l1 = 0.0f, ps0 = 0.0f, ps1 = 0.0f;
        for (uint32_t i0 = 0, round = 0; i0 < n; i0 += SW, ++round) {
            if (!mbarWait(&fullBar[round & 1u], (round >> 1) & 1u, p.err, kDevErrFullWait)) break;
            const uint32_t i1 = min(n, i0 + SW);
            for (uint32_t i = i0; i < i1; ++i) {
                const uint8_t *rec = record(i);
                const float *fac = reinterpret_cast<const float *>(rec + kRecF);
                const float *recP = reinterpret_cast<const float *>(rec + kRecP) + lane;
                const float *recX = reinterpret_cast<const float *>(rec + kRecX) + lane;
                float pv[2 * NR], xv[2 * NR];
#pragma unroll
                for (int r = 0; r < 2 * NR; ++r) pv[r] = recP[r * 32], xv[r] = recX[r * 32];
                if (*reinterpret_cast<const uint32_t *>(fac + 16) != 0u) {
                    const float2 al = *reinterpret_cast<const float2 *>(fac + 2 * t);
                    const float2 as = *reinterpret_cast<const float2 *>(fac + 8 + 2 * t);
                    l0 *= as.x, l1 *= as.y;
                    ps0 *= al.x, ps1 *= al.y;
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    l0 += pv[2 * r], l1 += pv[2 * r + 1];
                    ps0 += xv[2 * r], ps1 += xv[2 * r + 1];
                }
            }
            __syncwarp();
            if (lane == 0) mbarArrive(&emptyBar[round & 1u]);
        }
#pragma unroll
        for (int off = 4; off <= 16; off <<= 1) {
            l0 += __shfl_xor_sync(0xffffffffu, l0, off);
            l1 += __shfl_xor_sync(0xffffffffu, l1, off);
            ps0 += __shfl_xor_sync(0xffffffffu, ps0, off);
            ps1 += __shfl_xor_sync(0xffffffffu, ps1, off);
        }
        if (g == 0) {
            sEnd[16 + 2 * t] = l0, sEnd[17 + 2 * t] = l1;
            sEnd[24 + 2 * t] = ps0, sEnd[25 + 2 * t] = ps1;
        }
    }
    __syncthreads();
    float *scr = reinterpret_cast<float *>(smem);  // [8 heads][FoldScratch::kRow], then m[8], l[8]
    if (warp >= SW && warp < SW + VW) {
        // true accumulator = 2^24 * raw - 128 * sum(p*sv), then back from the E-scaled domain
        const float E = sEnd[8], c0 = 128.0f * sEnd[24 + 2 * t], c1 = 128.0f * sEnd[25 + 2 * t];
#pragma unroll
        for (int c = 0; c < 2 * CP; ++c) {
            const uint32_t d = (warp - SW) * (HD / 4) + 16 * c + 2 * g;
            *reinterpret_cast<float2 *>(scr + (2 * t) * FoldScratch<HD>::kRow + d) =
                    make_float2(fmaf(o[c][0], kI8Unscale, -c0) * E, fmaf(o[c][2], kI8Unscale, -c0) * E);
            *reinterpret_cast<float2 *>(scr + (2 * t + 1) * FoldScratch<HD>::kRow + d) =
                    make_float2(fmaf(o[c][1], kI8Unscale, -c1) * E, fmaf(o[c][3], kI8Unscale, -c1) * E);
        }
    } else if (warp == 0 && lane < 8u) {
        scr[FoldScratch<HD>::kM + lane] = sEnd[lane];
        scr[FoldScratch<HD>::kL + lane] = sEnd[16 + lane];
    }
    __syncthreads();
    FoldTarget f;
    f.out = p.out, f.pAcc = nullptr, f.pM = nullptr, f.pL = nullptr;
    f.numChunks = 1, f.slot = 0;
    f.firstHead = head0, f.nValid = nValid;
    f.direct = 1;
    f.qRot = nullptr, f.cosT = nullptr, f.sinT = nullptr, f.tableRow = 0;
    clusterFold<HD, 1, kThreads>(scr, f, threadIdx.x);
}

template <int HD, int MT>
static int launchStreams(DecodeI8Params prm, cudaStream_t st) {
    using L = I8StreamSmem<HD, MT>;
    auto kern = decodeI8StreamsKernel<HD, MT>;
    static ClusterSetup setup;
    const uint32_t *limits = nullptr;
    int rc = setupCluster(setup, kern, L::kWarps * 32, L::kTotal, &limits);
    if (rc != TC_OK) return rc;
    for (uint32_t cb = 0; cb < prm.group; cb += 8) {  // 8 q heads of a kv head per launch
        prm.colBase = cb;
        if (cb) prm.appendK = prm.appendV = nullptr;  // the row is in
        rc = launchDependent(kern, dim3(8, prm.nKV, 1), L::kWarps * 32, L::kTotal, st, 8, prm);
        if (rc != TC_OK) return rc;
    }
    return TC_OK;
}

int launchStreamsI8(DecodeI8Params prm, uint32_t hd, cudaStream_t st) {
    return hd == 256 ? launchStreams<256, 1>(prm, st) : launchStreams<128, 2>(prm, st);
}

}  // namespace tc
