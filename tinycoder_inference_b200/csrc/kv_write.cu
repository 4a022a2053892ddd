// kv_write.cu -- KV-cache writers: int8 quantise+append, f32/fp16 append with the
// optional NEOX rotation of K (and of Q in place), and RoPE(Q) alone.
//
// All three are pure streaming kernels (HBM-bound, a few hundred KB to a few MB
// per call): 128-bit loads and stores, no shared memory.  Arithmetic follows the reference element for element so the
// int8 bytes, scales and rotated values are bit-identical to
// kQ35QuantKV8 (include/gpu/GpuQwen35Kernels.hpp:586-637) and
// kStoreKVRope / kRoPEQ (include/gpu/GpuElementwiseKernels.hpp:425-483).
#include "tc_common.cuh"

namespace tc {

// ---------------------------------------------------------------------------
// int8 quantise + append
// ---------------------------------------------------------------------------
// One warp per (token, kv head).  hd is a multiple of 4 and at most 1024; lane l
// owns the float4 groups l, l+32, ...  amax is an exact max, so the reduction
// order is free; the division is IEEE (__fdiv_rn) and the rounding is
// round-half-even (__float2int_rn), which is what lrintf does under the default
// rounding mode.
template <int MAXV>
__global__ void __launch_bounds__(256)
kvQuantKernel(const float *__restrict__ k, const float *__restrict__ v, int8_t *__restrict__ k8,
              int8_t *__restrict__ v8, float *__restrict__ ks, float *__restrict__ vs, uint32_t tokens,
              uint32_t nKV, uint32_t hd, uint64_t dstTokenBase, uint64_t srcTokenBase,
              const uint32_t *__restrict__ devDstBase, uint32_t batchMode, uint64_t rowsPerSeq,
              const uint64_t *__restrict__ rowBase, const uint32_t *__restrict__ devLens, int32_t lenAdd,
              uint64_t maxRows, unsigned int *__restrict__ err) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t row = static_cast<uint64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const bool some = row < static_cast<uint64_t>(tokens) * nKV;
    const uint64_t t = row / nKV, h = row % nKV;
    const uint64_t src = ((srcTokenBase + t) * nKV + h) * hd;
    if (some && 32u * lane < hd) prefetchL2(k + src + 32u * lane), prefetchL2(v + src + 32u * lane);
    gridDepWait();  // (no gridDepLaunch: the next grid may request these rows ahead of its own wait)
    if (!some) return;
    if (devDstBase != nullptr) dstTokenBase = devDstBase[0];
    uint64_t dst = (dstTokenBase + t) * nKV + h;
    if (batchMode) {
        // source row t is the new token of sequence t; it goes behind that sequence's rows
        const uint64_t base = rowBase != nullptr ? rowBase[t] : t * rowsPerSeq;
        const uint64_t pos = devLens != nullptr ? static_cast<uint64_t>(static_cast<int64_t>(devLens[t]) + lenAdd)
                                                : dstTokenBase;
        dst = (base + pos) * nKV + h;
    }
    // A destination row read from device memory (a replayed graph past its window, a bad length)
    // is checked here, where it is known: the store is skipped and the error word says so.
    if (maxRows != 0 && dst >= maxRows * nKV) {
        if (lane == 0) atomicOr(err, kDevErrRowBound);
        return;
    }
    const uint32_t nvec = hd >> 2;
    float4 kx[MAXV], vx[MAXV];
    float mk = 0.0f, mv = 0.0f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
        const uint32_t i = lane + 32u * j;
        if (i < nvec) {
            kx[j] = __ldg(reinterpret_cast<const float4 *>(k + src) + i);
            vx[j] = __ldg(reinterpret_cast<const float4 *>(v + src) + i);
            mk = fmaxf(mk, fmaxf(fmaxf(fabsf(kx[j].x), fabsf(kx[j].y)), fmaxf(fabsf(kx[j].z), fabsf(kx[j].w))));
            mv = fmaxf(mv, fmaxf(fmaxf(fabsf(vx[j].x), fabsf(vx[j].y)), fmaxf(fabsf(vx[j].z), fabsf(vx[j].w))));
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        mk = fmaxf(mk, __shfl_xor_sync(0xffffffffu, mk, o));
        mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
    }
    const float sk = mk > 0.0f ? __fdiv_rn(mk, 127.0f) : 1.0f;
    const float sv = mv > 0.0f ? __fdiv_rn(mv, 127.0f) : 1.0f;
    if (lane == 0) {
        ks[dst] = sk;
        vs[dst] = sv;
    }
    auto q8 = [](float x, float s) -> uint32_t {
        int q = __float2int_rn(__fdiv_rn(x, s));
        q = q < -128 ? -128 : (q > 127 ? 127 : q);
        return static_cast<uint32_t>(q) & 0xffu;
    };
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
        const uint32_t i = lane + 32u * j;
        if (i < nvec) {
            const uint32_t pk = q8(kx[j].x, sk) | (q8(kx[j].y, sk) << 8) | (q8(kx[j].z, sk) << 16) |
                                (q8(kx[j].w, sk) << 24);
            const uint32_t pv = q8(vx[j].x, sv) | (q8(vx[j].y, sv) << 8) | (q8(vx[j].z, sv) << 16) |
                                (q8(vx[j].w, sv) << 24);
            reinterpret_cast<uint32_t *>(k8 + dst * hd)[i] = pk;
            reinterpret_cast<uint32_t *>(v8 + dst * hd)[i] = pv;
        }
    }
    __threadfence();  // in memory before the block's exit lets the next grid start
}

// ---------------------------------------------------------------------------
// f32 / fp16 append, optional rotation
// ---------------------------------------------------------------------------
// V consecutive elements of a row: loaded as floats, stored as KVT.
template <int V>
struct Vec {
    float x[V];
};
template <int V>
__device__ __forceinline__ Vec<V> loadVec(const float *p) {
    Vec<V> r;
    if constexpr (V == 4) {
        const float4 f = *reinterpret_cast<const float4 *>(p);
        r.x[0] = f.x, r.x[1] = f.y, r.x[2] = f.z, r.x[3] = f.w;
    } else {
        r.x[0] = *p;
    }
    return r;
}
template <int V>
__device__ __forceinline__ void storeVec(float *p, const Vec<V> &v) {
    if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(v.x[0], v.x[1], v.x[2], v.x[3]);
    else *p = v.x[0];
}
template <int V>
__device__ __forceinline__ void storeVec(__half *p, const Vec<V> &v) {
    if constexpr (V == 4) *reinterpret_cast<uint2 *>(p) = make_uint2(packHalf2(v.x[0], v.x[1]), packHalf2(v.x[2], v.x[3]));
    else *p = __float2half_rn(v.x[0]);
}

// A thread owns V rotation pairs (j .. j + V - 1 with their partners hd / 2 further on) of one head row of one
// token: rows [0, nHeads) of a token are q (rotated in place), then nKV rows of K (rotated, or verbatim without
// tables) and nKV rows of V (verbatim).  x0' = fmaf(x0, c, -(x1*s)), x1' = fmaf(x0, s, x1*c): the
// reference's form.  HBM-bound for prompts, launch-bound for a token (in a graph, with q of 28 heads rotated and 4 kv
// heads of 128 stored: 1 row 3.1 -> 1.3 us, 4096 rows 29.6 -> 18.7 us against a block per token with scalar loops).
// V = 4 wants 16-byte aligned rows and hd a multiple of 8, else V = 1.
template <typename KVT, int V>
__global__ void __launch_bounds__(256)
kvAppendKernel(float *__restrict__ q, const float *__restrict__ kSrc, const float *__restrict__ vSrc,
               KVT *__restrict__ kDst, KVT *__restrict__ vDst, uint32_t seqLen, uint32_t nHeads, uint32_t nKV, uint32_t hd,
               uint32_t cachePos, uint32_t ropePos, const uint32_t *__restrict__ devPos,
               const float *__restrict__ cosT, const float *__restrict__ sinT, uint32_t maxRows,
               unsigned int *__restrict__ err) {
    const uint32_t pairs = hd >> 1, perRow = pairs / V;
    const uint32_t rowsPerToken = nHeads + 2 * nKV;
    const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t rowIdx = idx / perRow;
    const bool some = rowIdx < static_cast<uint64_t>(seqLen) * rowsPerToken;
    const uint32_t j = static_cast<uint32_t>(idx - rowIdx * perRow) * V;
    const uint32_t s = static_cast<uint32_t>(rowIdx / rowsPerToken);
    uint32_t row = static_cast<uint32_t>(rowIdx - static_cast<uint64_t>(s) * rowsPerToken);
    const bool isQ = row < nHeads, isFirst = row == 0;
    if (!isQ) row -= nHeads;
    const bool isV = !isQ && row >= nKV;
    if (isV) row -= nKV;
    const float *src = isQ ? q + (static_cast<size_t>(s) * nHeads + row) * hd
                           : (isV ? vSrc : kSrc) + (static_cast<size_t>(s) * nKV + row) * hd;
    if (some) {
        prefetchLineOf(src + j, 4 * V);
        prefetchLineOf(src + j + pairs, 4 * V);
        if (cosT != nullptr && devPos == nullptr && isFirst) {  // (the token's table row once, not for q, K and V each)
            const size_t at = static_cast<size_t>(ropePos + s) * pairs + j;
            prefetchLineOf(cosT + at, 4 * V);
            prefetchLineOf(sinT + at, 4 * V);
        }
    }
    gridDepWait();
    gridDepLaunch();
    if (!some) return;
    if (devPos != nullptr) {
        cachePos = devPos[0];
        ropePos = devPos[0];
    }
    if (!isQ && maxRows != 0 && static_cast<uint64_t>(cachePos) + s >= maxRows) {
        // device-side position outside the window: no store, reported through the error word
        if (j == 0) atomicOr(err, kDevErrRowBound);
        return;
    }
    Vec<V> x0 = loadVec<V>(src + j), x1 = loadVec<V>(src + j + pairs);
    if (!isV && cosT != nullptr) {
        const size_t at = static_cast<size_t>(ropePos + s) * pairs + j;
        const Vec<V> c = loadVec<V>(cosT + at), sn = loadVec<V>(sinT + at);
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const float a = x0.x[i], b = x1.x[i];
            x0.x[i] = fmaf(a, c.x[i], -__fmul_rn(b, sn.x[i]));
            x1.x[i] = fmaf(a, sn.x[i], __fmul_rn(b, c.x[i]));
        }
    }
    if (isQ) {
        float *d = q + (static_cast<size_t>(s) * nHeads + row) * hd + j;
        storeVec<V>(d, x0);
        storeVec<V>(d + pairs, x1);
    } else {
        KVT *d = (isV ? vDst : kDst) + (static_cast<size_t>(cachePos + s) * nKV + row) * hd + j;
        storeVec<V>(d, x0);
        storeVec<V>(d + pairs, x1);
    }
}

// attnOut[s][h][e] *= 1/(1+exp(-gate)); gate is the second half of each head's
// fused q+gate row.  The reference evaluates the sigmoid with __expf.
// A thread owns V consecutive elements: HBM-bound for prompts (4096 rows of 16 x 256: 30.8 us, 6.5 TB/s), launch-bound
// for a token (1.3 us in a graph).  One block per token with a scalar loop and a division per element took 78.9 and
// 8.3 us.
template <int V>
__global__ void __launch_bounds__(256)
sigmoidGateKernel(float *__restrict__ attnOut, const float *__restrict__ qGate, uint64_t units, uint32_t hd) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint32_t perHead = hd / V;
    const uint64_t head = i / perHead;  // token x head
    const uint32_t e = static_cast<uint32_t>(i - head * perHead) * V;
    const float *gate = qGate + head * 2 * hd + hd + e;
    if (i < units) prefetchLineOf(gate, 4 * V);
    gridDepWait();
    gridDepLaunch();
    if (i >= units) return;
    const Vec<V> g = loadVec<V>(gate);
    Vec<V> x = loadVec<V>(attnOut + head * hd + e);
#pragma unroll
    for (int k = 0; k < V; ++k) x.x[k] *= 1.0f / (1.0f + __expf(-g.x[k]));
    storeVec<V>(attnOut + head * hd + e, x);
}

// Launch of kvAppendKernel: q (nullable) and K / V rows (nullable).
template <typename KVT>
static int launchAppend(float *q, const float *kSrc, const float *vSrc, void *kDst, void *vDst, uint32_t seqLen,
                        uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t cachePos, uint32_t ropePos,
                        const uint32_t *devPos, const float *cosT, const float *sinT, uint32_t maxRows, unsigned int *err,
                        cudaStream_t st) {
    uintptr_t align = 0;
    for (const void *p : {static_cast<const void *>(q), static_cast<const void *>(kSrc), static_cast<const void *>(vSrc),
                          static_cast<const void *>(kDst), static_cast<const void *>(vDst), static_cast<const void *>(cosT),
                          static_cast<const void *>(sinT)})
        align |= reinterpret_cast<uintptr_t>(p);
    const bool vec = (hd % 8u) == 0 && (align & 15u) == 0;
    if (q == nullptr || cosT == nullptr) nHeads = 0;
    if (kSrc == nullptr) nKV = 0;
    const uint64_t threads = static_cast<uint64_t>(seqLen) * (nHeads + 2ull * nKV) * (hd / 2 / (vec ? 4 : 1));
    const uint64_t blocks = (threads + 255) / 256;
    if (blocks == 0) return TC_OK;
    TC_REQUIRE(blocks <= 0x7fffffffull, TC_EUNSUPPORTED, "append: too many rows");
    auto kern = vec ? kvAppendKernel<KVT, 4> : kvAppendKernel<KVT, 1>;
    return launchDependent(kern, dim3(static_cast<uint32_t>(blocks)), 256, 0, st, 1, q, kSrc, vSrc,
                               static_cast<KVT *>(kDst), static_cast<KVT *>(vDst), seqLen, nHeads, nKV, hd, cachePos, ropePos,
                               devPos, cosT, sinT, maxRows, err);
}

// ---------------------------------------------------------------------------
// K and V store of a session zeroed
// ---------------------------------------------------------------------------
// One launch for both: what bounds a short call is the host's way to the GPU and back (the caller synchronises), and a memset
// each puts two launches into it.  clear() alone, memsets -> launch: 1 MB of K 12.2 -> 9.4 us, 16 MB 16.9 -> 14.4, 48 MB 26.0 -> 24.9,
// 64 MB 31.1 -> 30.7.  Longer ones are bound by HBM, which the memsets write at 7.2 TB/s and this loop at 6: 96 MB 40.8 -> 42.0,
// 256 MB 86 -> 97, 2 GB 596 -> 718.
constexpr size_t kClearLaunchBytes = size_t(64) << 20;  // of K, at most
__global__ void __launch_bounds__(256) kvClearKernel(uint4 *k, uint4 *v, size_t n) {
    gridDepWait();
    const size_t step = static_cast<size_t>(gridDim.x) * blockDim.x;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step) k[i] = zero, v[i] = zero;
}
// Whether both are the current device's own memory (0.15 us).  A memset takes the device from the address; a kernel would fault
// on memory of a device that is no peer of the current one.
static bool onCurrentDevice(const void *k, const void *v) {
    cudaPointerAttributes a, b;
    int dev = 0;
    const bool ok = cudaGetDevice(&dev) == cudaSuccess && cudaPointerGetAttributes(&a, k) == cudaSuccess &&
                    cudaPointerGetAttributes(&b, v) == cudaSuccess && a.type == cudaMemoryTypeDevice && a.device == dev &&
                    b.type == cudaMemoryTypeDevice && b.device == dev;
    if (!ok) cudaGetLastError();
    return ok;
}
int kvClear(void *k, void *v, size_t bytes, cudaStream_t st) {
    const size_t n = bytes / 16;
    if (n != 0 && bytes <= kClearLaunchBytes && ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | bytes) & 15u) == 0 &&
        onCurrentDevice(k, v)) {
        const size_t blocks = (n + 255) / 256, most = static_cast<size_t>(numSMs()) * 8;
        if (launchDependent(kvClearKernel, dim3(static_cast<uint32_t>(blocks < most ? blocks : most)), 256, 0, st, 1,
                            static_cast<uint4 *>(k), static_cast<uint4 *>(v), n) == TC_OK)
            return TC_OK;
        cudaGetLastError();  // (a stream of another device takes a memset, but no launch)
    }
    TC_CUDA_OK(cudaMemsetAsync(k, 0, bytes, st));
    TC_CUDA_OK(cudaMemsetAsync(v, 0, bytes, st));
    return TC_OK;
}

}  // namespace tc

extern "C" {

int tc_kv_quantize_i8(const float *k, const float *v, int8_t *k8, int8_t *v8, float *ks, float *vs,
                      uint32_t tokens, uint32_t nKV, uint32_t hd, uint64_t dstTokenBase,
                      uint64_t srcTokenBase, const uint32_t *devDstBase, uint64_t maxRows, tc_stream stream) {
    TC_REQUIRE(k && v && k8 && v8 && ks && vs, TC_EINVAL, "tc_kv_quantize_i8: null pointer");
    TC_REQUIRE(nKV > 0 && hd > 0 && (hd % 4u) == 0 && hd <= 1024, TC_EUNSUPPORTED,
               "tc_kv_quantize_i8: hd=%u must be a multiple of 4 and <= 1024", hd);
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15u) == 0 &&
                       ((reinterpret_cast<uintptr_t>(k8) | reinterpret_cast<uintptr_t>(v8)) & 3u) == 0,
               TC_EINVAL, "tc_kv_quantize_i8: k/v need 16-byte, k8/v8 4-byte alignment");
    if (tokens == 0) return TC_OK;
    if (devDstBase == nullptr && maxRows != 0 && dstTokenBase + tokens > maxRows) {
        tc::setError("tc_kv_quantize_i8: rows [%llu, %llu) pass the pool's %llu rows",
                     (unsigned long long) dstTokenBase, (unsigned long long) (dstTokenBase + tokens),
                     (unsigned long long) maxRows);
        return TC_ECONTEXT_FULL;
    }
    unsigned int *err = tc::devErrorWord();
    TC_REQUIRE(err != nullptr, TC_ECUDA, "tc_kv_quantize_i8: no device error word");
    const uint64_t rows = static_cast<uint64_t>(tokens) * nKV;
    const uint32_t warpsPerBlock = 8;
    const uint64_t blocks = (rows + warpsPerBlock - 1) / warpsPerBlock;
    TC_REQUIRE(blocks <= 0x7fffffffull, TC_EUNSUPPORTED, "tc_kv_quantize_i8: too many rows");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t nvec = hd / 4;
    auto kern = nvec <= 32 ? tc::kvQuantKernel<1> : (nvec <= 64 ? tc::kvQuantKernel<2> : tc::kvQuantKernel<8>);
    const uint64_t *noBase = nullptr;
    const uint32_t *noLens = nullptr;
    return tc::launchDependent(kern, dim3(static_cast<uint32_t>(blocks)), 256, 0, st, 1, k, v, k8, v8, ks, vs, tokens, nKV, hd,
                               dstTokenBase, srcTokenBase, devDstBase, 0u, uint64_t(0), noBase, noLens, 0, maxRows, err);
}

int tc_kv_quantize_i8_batch(const float *k, const float *v, int8_t *k8, int8_t *v8, float *ks, float *vs,
                            uint32_t batch, uint32_t nKV, uint32_t hd, uint64_t rowsPerSeq, const uint64_t *rowBase,
                            uint32_t pos, const uint32_t *lens, int32_t lenAdd, uint64_t totalRows, tc_stream stream) {
    TC_REQUIRE(k && v && k8 && v8 && ks && vs, TC_EINVAL, "tc_kv_quantize_i8_batch: null pointer");
    TC_REQUIRE(nKV > 0 && hd > 0 && (hd % 4u) == 0 && hd <= 1024, TC_EUNSUPPORTED,
               "tc_kv_quantize_i8_batch: hd=%u must be a multiple of 4 and <= 1024", hd);
    TC_REQUIRE(((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15u) == 0 &&
                       ((reinterpret_cast<uintptr_t>(k8) | reinterpret_cast<uintptr_t>(v8)) & 3u) == 0,
               TC_EINVAL, "tc_kv_quantize_i8_batch: k/v need 16-byte, k8/v8 4-byte alignment");
    if (batch == 0) return TC_OK;
    if (lens == nullptr && rowBase == nullptr && totalRows != 0 &&
        static_cast<uint64_t>(batch - 1) * rowsPerSeq + pos >= totalRows) {
        tc::setError("tc_kv_quantize_i8_batch: row %u of sequence %u passes the pool's %llu rows", pos, batch - 1,
                     (unsigned long long) totalRows);
        return TC_ECONTEXT_FULL;
    }
    unsigned int *err = tc::devErrorWord();
    TC_REQUIRE(err != nullptr, TC_ECUDA, "tc_kv_quantize_i8_batch: no device error word");
    const uint64_t rows = static_cast<uint64_t>(batch) * nKV;
    const uint32_t blocks = static_cast<uint32_t>((rows + 7) / 8);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t nvec = hd / 4;
    auto kern = nvec <= 32 ? tc::kvQuantKernel<1> : (nvec <= 64 ? tc::kvQuantKernel<2> : tc::kvQuantKernel<8>);
    const uint32_t *noDst = nullptr;
    return tc::launchDependent(kern, dim3(blocks), 256, 0, st, 1, k, v, k8, v8, ks, vs, batch, nKV, hd,
                               static_cast<uint64_t>(pos), uint64_t(0), noDst, 1u, rowsPerSeq, rowBase, lens, lenAdd,
                               totalRows, err);
}

static int appendCommon(float *q, const float *kSrc, const float *vSrc, void *kDst, void *vDst, int kvHalf,
                        uint32_t seqLen, uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t cachePos,
                        uint32_t ropePos, const uint32_t *devPos, const float *cosT, const float *sinT,
                        uint32_t maxRows, tc_stream stream, const char *who) {
    TC_REQUIRE(kSrc && vSrc && kDst && vDst, TC_EINVAL, "%s: null pointer", who);
    TC_REQUIRE(nKV > 0 && hd > 0 && (hd % 2u) == 0, TC_EUNSUPPORTED, "%s: hd=%u must be even", who, hd);
    TC_REQUIRE((cosT == nullptr) == (sinT == nullptr), TC_EINVAL, "%s: cos and sin tables come together", who);
    if (seqLen == 0) return TC_OK;
    if (devPos == nullptr && maxRows != 0 &&
        static_cast<uint64_t>(cachePos) + seqLen > static_cast<uint64_t>(maxRows)) {
        tc::setError("%s: rows [%u, %llu) pass the window of %u rows", who, cachePos,
                     (unsigned long long) cachePos + seqLen, maxRows);
        return TC_ECONTEXT_FULL;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned int *err = tc::devErrorWord();
    TC_REQUIRE(err != nullptr, TC_ECUDA, "%s: no device error word", who);
    return kvHalf ? tc::launchAppend<__half>(q, kSrc, vSrc, kDst, vDst, seqLen, nHeads, nKV, hd, cachePos, ropePos, devPos, cosT,
                                         sinT, maxRows, err, st)
                  : tc::launchAppend<float>(q, kSrc, vSrc, kDst, vDst, seqLen, nHeads, nKV, hd, cachePos, ropePos, devPos, cosT,
                                        sinT, maxRows, err, st);
}

int tc_kv_append(const float *kSrc, const float *vSrc, void *kDst, void *vDst, int kvHalf, uint32_t seqLen,
                 uint32_t nKV, uint32_t hd, uint32_t cachePos, const uint32_t *devPos, uint32_t maxRows,
                 tc_stream stream) {
    return appendCommon(nullptr, kSrc, vSrc, kDst, vDst, kvHalf, seqLen, 0, nKV, hd, cachePos, 0, devPos,
                        nullptr, nullptr, maxRows, stream, "tc_kv_append");
}

int tc_kv_append_rope(float *q, const float *kSrc, const float *vSrc, void *kDst, void *vDst, int kvHalf,
                      uint32_t seqLen, uint32_t nHeads, uint32_t nKV, uint32_t hd, uint32_t cachePos,
                      uint32_t ropePos, const uint32_t *devPos, const float *cosT, const float *sinT,
                      uint32_t maxRows, tc_stream stream) {
    TC_REQUIRE(cosT && sinT, TC_EINVAL, "tc_kv_append_rope: cos/sin tables are required");
    return appendCommon(q, kSrc, vSrc, kDst, vDst, kvHalf, seqLen, nHeads, nKV, hd, cachePos, ropePos, devPos,
                        cosT, sinT, maxRows, stream, "tc_kv_append_rope");
}

int tc_rope_q(float *q, const float *cosT, const float *sinT, uint32_t seqLen, uint32_t nHeads, uint32_t hd,
              uint32_t pos, const uint32_t *devPos, tc_stream stream) {
    TC_REQUIRE(q && cosT && sinT, TC_EINVAL, "tc_rope_q: null pointer");
    TC_REQUIRE(hd > 0 && (hd % 2u) == 0, TC_EUNSUPPORTED, "tc_rope_q: hd=%u must be even", hd);
    if (seqLen == 0) return TC_OK;
    return tc::launchAppend<float>(q, nullptr, nullptr, nullptr, nullptr, seqLen, nHeads, 0, hd, 0, pos, devPos, cosT, sinT, 0u,
                               nullptr, static_cast<cudaStream_t>(stream));
}

int tc_attn_sigmoid_gate(float *attnOut, const float *qGate, uint32_t seqLen, uint32_t nHeads, uint32_t hd,
                         tc_stream stream) {
    TC_REQUIRE(attnOut && qGate, TC_EINVAL, "tc_attn_sigmoid_gate: null pointer");
    if (seqLen == 0) return TC_OK;
    const bool vec = (hd % 4u) == 0 && ((reinterpret_cast<uintptr_t>(attnOut) | reinterpret_cast<uintptr_t>(qGate)) & 15u) == 0;
    const uint64_t units = static_cast<uint64_t>(seqLen) * nHeads * (hd / (vec ? 4u : 1u));
    if (units == 0) return TC_OK;
    TC_REQUIRE((units + 255) / 256 <= 0x7fffffffull, TC_EUNSUPPORTED, "tc_attn_sigmoid_gate: too many rows");
    return tc::launchDependent(vec ? tc::sigmoidGateKernel<4> : tc::sigmoidGateKernel<1>,
                               dim3(static_cast<uint32_t>((units + 255) / 256)), 256, 0, static_cast<cudaStream_t>(stream), 1,
                               attnOut, qGate, units, hd);
}

}  // extern "C"
