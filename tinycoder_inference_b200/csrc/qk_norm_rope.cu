// qk_norm_rope.cu -- the step in front of attention in the hybrid (gated) models: per-head
// RMSNorm of Q and K fused with the partial NEOX rotation by the MRoPE tables.
//
// What it replaces: kQ35QNormRoPE and kQ35KNormRoPE (include/gpu/GpuQwen35Kernels.hpp:55-137),
// launched back to back in front of the KV store
// (src/cpp/core/cuda/forward/GPUComputeForward.cu:1330-1337):
//   rms = rsqrt(sum(x^2) / hd + 1e-6);  y_j = x_j * rms * w_j;
//   j < nDims/2:  out_j = fma(y_j, c_j, -y_{j+h} * s_j),  out_{j+h} = fma(y_j, s_j, y_{j+h} * c_j)
//   j >= nDims:   out_j = y_j                                   (h = nDims/2, tables [pos][h])
// Q is read from the projection's [token][head][2*hd] rows (q then gate) and written out of
// place as [token][head][hd]; K is normalised in place.
//
// One launch does both, one WARP per (token, head) slice with everything in registers (the
// reference uses a 128-thread block and a shared-memory tree per slice).  The sum of squares
// is folded in the reference's order -- element j belongs to thread j mod 128 of its block,
// threads are folded 64, 32, ..., 1 apart -- so the normaliser, and with it every output, is
// bit-identical: a lane carries the four "threads" lane, lane+32, lane+64, lane+96.
#include "tc_common.cuh"

namespace tc {

constexpr int kNormMaxPer = 4;  // elements per reference thread: hd <= 512

// What bounds it: latency for a token (18 slices of a 16 + 2 head model), HBM for prompts.  Every load of a lane --
// its elements, the norm weights, the table row -- is requested before the first one is used, and with the
// rotated half a multiple of 32 (HB = half / 32) an element's partner sits in the same lane, HB registers further on.
// (16 + 2 heads of 256, in a graph: 1 row 1.3 us, 333 rows 2.8, 4096 rows 26.4; with partners, weights and table
// entries fetched behind the reduction 3.2, 6.0 and 50.0.)  HB = 0: any other half; partners come from the row
// again (it is in L1).  PER: 128-element groups of a slice.
template <int PER, int HB>
__global__ void __launch_bounds__(256)
qkNormRopeKernel(const float *__restrict__ qIn, uint32_t qInStride, float *qOut, float *k,
                 const float *__restrict__ wq, const float *__restrict__ wk, uint32_t hd, uint32_t nDims,
                 uint32_t nHeads, uint32_t nKV, uint32_t seqLen, uint32_t pos, const uint32_t *__restrict__ devPos,
                 const float *__restrict__ cosT, const float *__restrict__ sinT) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t slices = (qIn ? nHeads : 0u) + (k ? nKV : 0u);
    const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const bool some = idx < static_cast<uint64_t>(seqLen) * slices;
    const uint32_t s = static_cast<uint32_t>(idx / slices);
    uint32_t h = static_cast<uint32_t>(idx % slices);
    const bool isQ = qIn != nullptr && h < nHeads, isFirst = h == 0u;
    if (!isQ && qIn != nullptr) h -= nHeads;
    const float *rp = isQ ? qIn + (static_cast<uint64_t>(s) * nHeads + h) * qInStride
                          : k + (static_cast<uint64_t>(s) * nKV + h) * hd;
    float *op = isQ ? qOut + (static_cast<uint64_t>(s) * nHeads + h) * hd : k + (static_cast<uint64_t>(s) * nKV + h) * hd;
    const float *w = isQ ? wq : wk;
    if (some) {
        if (32u * lane < hd) {
            prefetchL2(rp + 32u * lane);
            if (s == 0u && h == 0u) prefetchL2(w + 32u * lane);
        }
        if (devPos == nullptr && isFirst && 64u * lane < nDims) {  // (the token's table row once, not for q and K each)
            const uint64_t at = static_cast<uint64_t>(pos + s) * (nDims / 2) + 32u * lane;
            prefetchL2(cosT + at), prefetchL2(sinT + at);
        }
    }
    gridDepWait();
    gridDepLaunch();
    if (!some) return;

    // element e of a lane is j = lane + 32 e: e = i + 4 kk is the kk-th element of reference thread lane + 32 i
    constexpr int E = 4 * PER;
    float x[E], wv[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t j = lane + 32u * e;
        x[e] = j < hd ? rp[j] : 0.0f;
        wv[e] = j < hd ? w[j] : 0.0f;
    }
    const uint32_t p = (devPos != nullptr ? devPos[0] : pos) + s;
    const uint32_t half = HB ? HB * 32u : nDims / 2;
    const float *c = cosT + static_cast<uint64_t>(p) * half;
    const float *sn = sinT + static_cast<uint64_t>(p) * half;
    constexpr int kHalfRegs = HB ? HB : 1;
    float cv[kHalfRegs], sv[kHalfRegs];
    if (HB) {
#pragma unroll
        for (int e = 0; e < kHalfRegs; ++e) cv[e] = c[lane + 32u * e], sv[e] = sn[lane + 32u * e];
    }
    float a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        a[i] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < PER; ++kk)
            if (lane + 32u * i + 128u * kk < hd) a[i] = fmaf(x[i + 4 * kk], x[i + 4 * kk], a[i]);
    }
    float sum = (a[0] + a[2]) + (a[1] + a[3]);  // threads 64 apart, then 32 apart
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    sum = __shfl_sync(0xffffffffu, sum, 0);
    const float rms = rsqrtf(sum / static_cast<float>(hd) + 1e-6f);
    float y[E];
#pragma unroll
    for (int e = 0; e < E; ++e) y[e] = x[e] * rms * wv[e];
    if (HB) {
#pragma unroll
        for (int e = 0; e < HB && e + HB < E; ++e) {
            const float y0 = y[e], y1 = y[e + HB];
            y[e] = fmaf(y0, cv[e], -y1 * sv[e]);
            y[e + HB] = fmaf(y0, sv[e], y1 * cv[e]);
        }
    } else {
        // (K is rotated in place: every read happens before the first write)
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint32_t j = lane + 32u * e;
            if (j >= hd) continue;
            if (j < half) {
                const float y1 = rp[j + half] * rms * w[j + half];
                y[e] = fmaf(y[e], c[j], -y1 * sn[j]);
            } else if (j < nDims) {
                const uint32_t j0 = j - half;
                const float y0 = rp[j0] * rms * w[j0];
                y[e] = fmaf(y0, sn[j0], y[e] * c[j0]);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t j = lane + 32u * e;
        if (j < hd) op[j] = y[e];
    }
}

}  // namespace tc

extern "C" int tc_qk_norm_rope(const float *qIn, uint32_t qInStride, float *qOut, float *k, const float *wq,
                               const float *wk, uint32_t hd, uint32_t nDims, uint32_t nHeads, uint32_t nKV,
                               uint32_t seqLen, uint32_t pos, const uint32_t *devPos, const float *cosT,
                               const float *sinT, uint32_t tableRows, tc_stream stream) {
    TC_REQUIRE(cosT && sinT, TC_EINVAL, "tc_qk_norm_rope: null table");
    TC_REQUIRE((qIn == nullptr) == (qOut == nullptr), TC_EINVAL, "tc_qk_norm_rope: q input and output go together");
    TC_REQUIRE(qIn != nullptr || k != nullptr, TC_EINVAL, "tc_qk_norm_rope: nothing to do");
    TC_REQUIRE((qIn == nullptr || wq != nullptr) && (k == nullptr || wk != nullptr), TC_EINVAL,
               "tc_qk_norm_rope: missing norm weight");
    TC_REQUIRE(hd >= 2 && hd <= 128u * tc::kNormMaxPer, TC_EUNSUPPORTED, "tc_qk_norm_rope: head_dim %u (max %u)", hd,
               128u * tc::kNormMaxPer);
    TC_REQUIRE(nDims <= hd && (nDims % 2u) == 0, TC_EINVAL, "tc_qk_norm_rope: %u rotated dims of %u", nDims, hd);
    TC_REQUIRE(qIn == nullptr || qInStride >= hd, TC_EINVAL, "tc_qk_norm_rope: q row stride %u < head_dim", qInStride);
    // in place on the same buffer the rotation would read partners it has already overwritten
    TC_REQUIRE(qIn == nullptr || static_cast<const void *>(qIn) != static_cast<const void *>(qOut), TC_EINVAL,
               "tc_qk_norm_rope: q must be written out of place");
    if (seqLen == 0) return TC_OK;
    if (devPos == nullptr && static_cast<uint64_t>(pos) + seqLen > tableRows) {
        tc::setError("tc_qk_norm_rope: positions [%u, %llu) pass the %u table rows", pos,
                     (unsigned long long) pos + seqLen, tableRows);
        return TC_ECONTEXT_FULL;
    }
    const uint64_t warps = static_cast<uint64_t>(seqLen) * ((qIn ? nHeads : 0u) + (k ? nKV : 0u));
    const uint32_t blocks = static_cast<uint32_t>((warps + 7) / 8);
    // partners in the lane when the rotated half is 1, 2 or 4 x 32 elements (64, 128 or 256 rotated dims)
    const uint32_t hb = nDims == 64 ? 1u : (nDims == 128 ? 2u : (nDims == 256 ? 4u : 0u));
    const uint32_t per = hd <= 128 ? 1u : (hd <= 256 ? 2u : 4u);
    using Kern = decltype(&tc::qkNormRopeKernel<1, 0>);
    static const Kern kerns[3][4] = {
            {tc::qkNormRopeKernel<1, 0>, tc::qkNormRopeKernel<1, 1>, tc::qkNormRopeKernel<1, 2>, tc::qkNormRopeKernel<1, 0>},
            {tc::qkNormRopeKernel<2, 0>, tc::qkNormRopeKernel<2, 1>, tc::qkNormRopeKernel<2, 2>, tc::qkNormRopeKernel<2, 4>},
            {tc::qkNormRopeKernel<4, 0>, tc::qkNormRopeKernel<4, 1>, tc::qkNormRopeKernel<4, 2>, tc::qkNormRopeKernel<4, 4>}};
    const Kern kern = kerns[per == 1 ? 0 : (per == 2 ? 1 : 2)][hb == 4 ? 3 : hb];
    return tc::launchDependent(kern, dim3(blocks), 256, 0, static_cast<cudaStream_t>(stream), 1, qIn, qInStride, qOut, k, wq, wk,
                               hd, nDims, nHeads, nKV, seqLen, pos, devPos, cosT, sinT);
}
