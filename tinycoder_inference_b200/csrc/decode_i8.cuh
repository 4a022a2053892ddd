// decode_i8.cuh -- what the mma.sync kernels over the int8 store share (decode_i8.cu, decode_i8_streams.cu): the launch
// parameters, a head group's query fragments, a tile's scores.
#pragma once

#include "decode_cluster.cuh"

namespace tc {

struct DecodeI8Params {
    const float *q;
    float *out;
    const float *ks, *vs;
    float *pAcc, *pM, *pL;
    const uint32_t *devLens;     // nullable
    const uint64_t *devRowBase;  // nullable
    uint64_t rowsPerSeq, totalRows;
    uint32_t lenHost, lenAdd;
    uint32_t nHeads, nKV, group;
    uint32_t colBase;  // decode: the 8 MMA columns are q heads colBase .. colBase + 7 of the kv head
    uint32_t chunkTokens, numChunks;
    const float *appendK, *appendV;  // nullable: [batch][nKV][hd] rows to quantise into row len - 1 first
    uint32_t *k8w, *v8w;             // the pools
    F32Mirror mir;                   // and the f32 store that gets it verbatim
    // rows mode (causal prefill over the store): the 8 MMA columns of a CTA are 8
    // consecutive query rows of ONE q head instead of the q heads of one kv head;
    // row s attends pool rows [0, cachePos + s].  grid = (1, nHeads, ceil(qRows / 8)).
    uint32_t qRows, cachePos;
    const uint32_t *devPos;
    float invSqrt;
    int directOut;
    unsigned int *err;
};

// One sequence, no partial buffers, the accumulation order of the causal kernel (decode_i8_streams.cu).
int launchStreamsI8(DecodeI8Params prm, uint32_t hd, cudaStream_t st);

#ifdef __CUDACC__

// How far the running reference point of the softmax may lag behind the true
// maximum (log2 units) before the accumulators are rescaled.  p stays <= 2^8.
constexpr float kLazyLog2 = 8.0f;

// K and V bytes enter the products as fp16 subnormals: 2^-24 of their value.
constexpr float kI8Unscale = 16777216.0f;

// The query vectors of up to eight columns as MMA operands, and the constants of the two score columns (2t, 2t + 1) that a
// thread holds.
template <int HD>
struct I8Query {
    uint32_t hi[HD / 16][2], lo[HD / 16][2];
    float cs0, cs1;    // log2-domain scale
    float off0, off1;  // what the offset of the K bytes adds
};

// qp: the vector of column g = lane / 4 (any valid address when the column is not).
// q fragments for head column n = g of this kv head's group: power-of-two
// normalised, split into fp16 hi + lo, laid out as the B operand whose k
// slots follow the byte order ldmatrix hands out (dims 16c + 4t + {0..3}).
// behind() is called once the loads are on their way.
template <int HD, typename Behind>
__device__ __forceinline__ void i8LoadQuery(I8Query<HD> &f, const float *qp, bool valid, float invSqrt, uint32_t lane, Behind behind) {
    constexpr int NC = HD / 16;
    const uint32_t t = lane & 3u;
    float headScale, headOff;
    {
        float4 qv[NC];
        float amax = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; ++c)
            qv[c] = valid ? __ldg(reinterpret_cast<const float4 *>(qp + 16 * c + 4 * t)) : make_float4(0.f, 0.f, 0.f, 0.f);
        behind();
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(qv[c].x), fabsf(qv[c].y)), fmaxf(fabsf(qv[c].z), fabsf(qv[c].w))));
        }
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        int e = static_cast<int>((__float_as_uint(amax) >> 23) & 0xffu) - 127;  // floor(log2 amax)
        e = amax > 0.0f ? max(-100, min(100, e)) : 0;
        const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);  // 2^-e
        const float up = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);    // 2^e
        headScale = invSqrt * up * kLog2e;
        float qsum = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            float h0, l0, h1, l1, h2, l2, h3, l3;
            splitHalf(qv[c].x * down, h0, l0);
            splitHalf(qv[c].y * down, h1, l1);
            splitHalf(qv[c].z * down, h2, l2);
            splitHalf(qv[c].w * down, h3, l3);
            f.hi[c][0] = packHalf2(h0, h1);
            f.hi[c][1] = packHalf2(h2, h3);
            f.lo[c][0] = packHalf2(l0, l1);
            f.lo[c][1] = packHalf2(l2, l3);
            // the column sum the MMA really sees: the fp16-rounded parts
            const __half2 a = *reinterpret_cast<__half2 *>(&f.lo[c][0]), bb = *reinterpret_cast<__half2 *>(&f.lo[c][1]);
            qsum += (h0 + __low2float(a)) + (h1 + __high2float(a)) + (h2 + __low2float(bb)) + (h3 + __high2float(bb));
        }
        qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
        qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
        headOff = 128.0f * qsum;  // K bytes enter the MMA as x + 128
    }
    // score columns of this thread are heads 2t and 2t+1: fetch their constants
    f.cs0 = __shfl_sync(0xffffffffu, headScale, (2 * t) * 4);
    f.cs1 = __shfl_sync(0xffffffffu, headScale, (2 * t + 1) * 4);
    f.off0 = __shfl_sync(0xffffffffu, headOff, (2 * t) * 4);
    f.off1 = __shfl_sync(0xffffffffu, headOff, (2 * t + 1) * 4);
}

// The same by all NW warps of a block together, through `share` in its shared memory: a warp takes HD / (16 NW) of the 16-dim
// groups, then everybody reads all fragments.  (One warp alone spends 700 instructions on the 64 dims of a lane at head_dim
// 256, and eight warps of an SM doing that for themselves 1.2 us of a decode call.)  Bit for bit what i8LoadQuery gives: the
// sums keep its order.  Called by all threads of those warps; BAR: a named barrier for them (0: they are the block).
template <int HD, int NW>
struct I8QueryShare {
    static constexpr int NC = HD / 16;
    static constexpr int kFrag = 0;                     // [NC][32 lanes] uint4: hi, lo
    static constexpr int kSum = kFrag + NC * 512;       // [NC][32] sums of the rounded parts
    static constexpr int kMax = kSum + NC * 128;        // [NW][32] maxima
    static constexpr int kBytes = kMax + NW * 128;
    static_assert(NC % NW == 0, "whole groups per warp");
};
template <int HD, int NW, int BAR, typename Behind>
__device__ __forceinline__ void i8LoadQueryShared(I8Query<HD> &f, uint8_t *share, const float *qp, bool valid, float invSqrt,
                                                  uint32_t warp, uint32_t lane, Behind behind) {
    using S = I8QueryShare<HD, NW>;
    constexpr int NC = S::NC, N = NC / NW;
    const uint32_t t = lane & 3u;
    uint4 *frag = reinterpret_cast<uint4 *>(share + S::kFrag) + lane;
    float *sum = reinterpret_cast<float *>(share + S::kSum) + lane, *top = reinterpret_cast<float *>(share + S::kMax) + lane;
    float4 qv[N];
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int c = warp * N + i;
        qv[i] = valid ? *reinterpret_cast<const float4 *>(qp + 16 * c + 4 * t) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    behind();
#pragma unroll
    for (int i = 0; i < N; ++i)
        amax = fmaxf(amax, fmaxf(fmaxf(fabsf(qv[i].x), fabsf(qv[i].y)), fmaxf(fabsf(qv[i].z), fabsf(qv[i].w))));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    top[warp * 32] = amax;
    auto sync = [] {
        if (BAR == 0) __syncthreads();
        else namedBarSync(BAR, NW * 32);
    };
    sync();
#pragma unroll
    for (int w = 0; w < NW; ++w) amax = fmaxf(amax, top[w * 32]);
    int e = static_cast<int>((__float_as_uint(amax) >> 23) & 0xffu) - 127;  // floor(log2 amax)
    e = amax > 0.0f ? max(-100, min(100, e)) : 0;
    const float down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);  // 2^-e
    const float up = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);    // 2^e
    const float headScale = invSqrt * up * kLog2e;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int c = warp * N + i;
        float h0, l0, h1, l1, h2, l2, h3, l3;
        splitHalf(qv[i].x * down, h0, l0);
        splitHalf(qv[i].y * down, h1, l1);
        splitHalf(qv[i].z * down, h2, l2);
        splitHalf(qv[i].w * down, h3, l3);
        uint4 x = make_uint4(packHalf2(h0, h1), packHalf2(h2, h3), packHalf2(l0, l1), packHalf2(l2, l3));
        frag[c * 32] = x;
        const __half2 a = *reinterpret_cast<__half2 *>(&x.z), bb = *reinterpret_cast<__half2 *>(&x.w);
        sum[c * 32] = (h0 + __low2float(a)) + (h1 + __high2float(a)) + (h2 + __low2float(bb)) + (h3 + __high2float(bb));
    }
    sync();
    float qsum = 0.0f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const uint4 x = frag[c * 32];
        f.hi[c][0] = x.x, f.hi[c][1] = x.y, f.lo[c][0] = x.z, f.lo[c][1] = x.w;
        qsum += sum[c * 32];
    }
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
    const float headOff = 128.0f * qsum;
    f.cs0 = __shfl_sync(0xffffffffu, headScale, (2 * t) * 4);
    f.cs1 = __shfl_sync(0xffffffffu, headScale, (2 * t + 1) * 4);
    f.off0 = __shfl_sync(0xffffffffu, headOff, (2 * t) * 4);
    f.off1 = __shfl_sync(0xffffffffu, headOff, (2 * t + 1) * 4);
}

// log2-domain scores of a tile (16 MT tokens at kTile, their K scales at sK) against the eight columns: sc[r][0 / 1] is
// token g + 8 r against column 2t / 2t + 1; tokens tokBase + 8 r >= len0 / len1 are masked out.
template <int HD, int MT>
__device__ __forceinline__ void i8Scores(const I8Query<HD> &f, uint32_t kTile, const float *sK, uint32_t tokBase, uint32_t len0,
                                         uint32_t len1, uint32_t lane, float (&sc)[2 * MT][2]) {
    constexpr int NC = HD / 16, NR = 2 * MT;
    const uint32_t g = lane >> 2;
    const uint32_t lr = (lane & 7u) + ((lane >> 3) & 1u) * 8u;  // ldmatrix row this lane addresses
    const uint32_t lco = lane >> 4;                             // and which chunk of the pair
    const uint32_t lmOff = lr * 128;
    bool vl0[NR], vl1[NR];
    float skr[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {  // rows g, g+8, ... of this warp's tokens
        vl0[r] = tokBase + 8 * r < len0;
        vl1[r] = tokBase + 8 * r < len1;
        skr[r] = sK[g + 8 * r];
    }

    // ---- S^T = K . Q^T, two 16-token tiles x 8 heads ----
    float sh[MT][4], sl[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < 4; ++i) sh[mt][i] = sl[mt][i] = 0.0f;
#pragma unroll
    for (int cp = 0; cp < NC / 2; ++cp) {
        const uint32_t sw = (((2 * (cp & 3) + lco) ^ (lr & 7u)) << 4) + (cp >> 2) * (16 * MT * 128);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            uint32_t r0, r1, r2, r3;
            ldmatrixX4(r0, r1, r2, r3, kTile + mt * 2048 + lmOff + sw);
            r0 ^= 0x80808080u;
            r1 ^= 0x80808080u;
            r2 ^= 0x80808080u;
            r3 ^= 0x80808080u;
            {
                const uint32_t a0 = subnormalPair<0x4140>(r0), a1 = subnormalPair<0x4140>(r1),
                               a2 = subnormalPair<0x4342>(r0), a3 = subnormalPair<0x4342>(r1);
                mmaF16(sh[mt], a0, a1, a2, a3, f.hi[2 * cp][0], f.hi[2 * cp][1]);
                mmaF16(sl[mt], a0, a1, a2, a3, f.lo[2 * cp][0], f.lo[2 * cp][1]);
            }
            {
                const uint32_t a0 = subnormalPair<0x4140>(r2), a1 = subnormalPair<0x4140>(r3),
                               a2 = subnormalPair<0x4342>(r2), a3 = subnormalPair<0x4342>(r3);
                mmaF16(sh[mt], a0, a1, a2, a3, f.hi[2 * cp + 1][0], f.hi[2 * cp + 1][1]);
                mmaF16(sl[mt], a0, a1, a2, a3, f.lo[2 * cp + 1][0], f.lo[2 * cp + 1][1]);
            }
        }
    }
    // log2-domain scores: undo the 2^-24 of the subnormal operand and the +128 offset,
    // apply the row's K scale; rows past the range are masked out
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int r = 2 * mt + hf;
            const float d0 = fmaf(sh[mt][2 * hf] + sl[mt][2 * hf], kI8Unscale, -f.off0);
            const float d1 = fmaf(sh[mt][2 * hf + 1] + sl[mt][2 * hf + 1], kI8Unscale, -f.off1);
            sc[r][0] = vl0[r] ? d0 * (skr[r] * f.cs0) : -INFINITY;
            sc[r][1] = vl1[r] ? d1 * (skr[r] * f.cs1) : -INFINITY;
        }
    }
}

#endif  // __CUDACC__

}  // namespace tc
