// tc_common.cuh -- sm_100a device helpers shared by the attention kernels:
// mbarrier, TMA (cp.async.bulk.tensor), cp.async, ldmatrix, movmatrix, mma.sync,
// int8 -> fp16 conversion, plus the host-side error plumbing of the C ABI.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/tc_attn.h"

namespace tc {

constexpr float kLog2e = 1.4426950408889634f;  // same constant as the reference (GpuCommon.hpp:77)
constexpr float kNegBig = -1e30f;              // initial running max of the GPU kernels

// Device-side error word: a kernel that gives up on a bounded wait ORs a code in
// and returns; tc_device_status() reads and clears it.
enum : uint32_t {
    kDevErrFullWait = 1u,   // consumer waited too long for a TMA stage
    kDevErrEmptyWait = 2u,  // producer waited too long for a free stage
    kDevErrMmaWait = 4u,    // waited too long for a tcgen05 commit
    kDevErrTmemAlloc = 8u,
    kDevErrMergeWait = 16u,  // a block waited too long for the partials of another rank
    kDevErrRowBound = 32u,   // a KV writer was handed a device-side position outside its pool: store skipped
};
// The word lives in one translation unit; kernels receive its device address as
// an argument (devErrorWord(), resolved once per device).
unsigned int *devErrorWord();

// ---- host-side error reporting ---------------------------------------------
void setError(const char *fmt, ...);
int cudaFail(cudaError_t e, const char *what);
#define TC_CUDA_OK(expr)                                    \
    do {                                                    \
        cudaError_t _e = (expr);                            \
        if (_e != cudaSuccess) return tc::cudaFail(_e, #expr); \
    } while (0)
#define TC_REQUIRE(cond, code, ...)      \
    do {                                 \
        if (!(cond)) {                   \
            tc::setError(__VA_ARGS__);   \
            return (code);               \
        }                                \
    } while (0)

int numSMs();

// Tensor-map factory (driver entry point resolved through the runtime, cached
// per (pointer, shape)).  All maps are uint8 / 2-byte / 4-byte element tiles.
struct TensorMapKey {
    const void *base;
    uint64_t dims[4];
    uint64_t strides[3];  // bytes, dims 1..3
    uint32_t box[4];
    uint32_t rank, elemBytes, swizzle;  // swizzle: 0 none, 1 32B, 2 64B, 3 128B
    uint32_t pad_;                      // keeps the struct free of implicit padding (it is memcmp'd)
};
int getTensorMap(const TensorMapKey &key, CUtensorMap *out);

#ifdef __CUDACC__

// Launch under programmatic dependent launch: the grid may be scheduled while the one in front of it drains, so
// the kernel has to call gridDepWait() before it touches anything that grid may have written or may still read --
// every kernel launched through here does so first thing (hints towards L2 may go ahead of it), but for the int8 decode at head_dim 128 under
// TC_DECODE_PDL, which requests rows of its pool that the caller calls old (prefetchRows) ahead of it.  Where the others
// call gridDepLaunch() decides what such a launch may find unfinished:
//   * after the wait, so that the kernels ahead of theirs are complete;
//   * a kernel that writes int8 rows of head_dim 128 (nothing else is read ahead of a wait), not before those are in
//     memory: kvQuantKernel by its exit, a decode kernel that takes the new row along behind that row's store.  The rows
//     launch of a prompt may let the next grid in sooner: that is the attention launch, which waits before it does.
// So a row written by any call without TC_DECODE_PDL is in memory before a call behind it can look.  (In stream order a dependent launch takes 3.1 - 3.7 us on
// B200, like this 2.0; as nodes of a graph 1.2 and 0.8.)  cluster: blocks per cluster along x.
template <typename... P, typename... A>
int launchDependent(void (*kern)(P...), dim3 grid, uint32_t threads, size_t smem, cudaStream_t st, uint32_t cluster,
                    const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    TC_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, args...));
    return TC_OK;
}

// What a kernel is handed -- q, new rows, gates, rotation tables -- towards L2 ahead of its dependency wait: where DRAM still holds
// it, a chain of short launches waited for it at each of them.  Right at any time: it is a hint, and what a kernel in flight
// still writes is read after the wait.  (Each line once: the norm weights asked for by every warp of a 333-row launch cost 6 us.)
// Eight layers of 16 / 2 / 256 behind 16383 int8 rows, norm and gate included, 140.0 -> 134.2 us (as a graph 121.7 -> 115.8); four of 28 / 4 / 128 behind 8191 fp16
// rows 30.0 -> 29.5; four of a 333-row prompt of 16 / 2 / 256 101.3 -> 96.8.
__device__ __forceinline__ void prefetchL2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// (`bytes` and the address multiples of 16)
__device__ __forceinline__ void prefetchBulkL2(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// ... of a line of 128 bytes whose first bytes this thread reads (`n` of them at `p`)
__device__ __forceinline__ void prefetchLineOf(const void *p, uint32_t n) {
    if ((reinterpret_cast<uintptr_t>(p) & 127u) < n) prefetchL2(p);
}

// ---- mbarrier ----------------------------------------------------------------
constexpr uint32_t kMbarSuspendNs = 20000u;  // upper bound of one hardware-parked poll
__device__ __forceinline__ uint32_t smemAddr(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbarInit(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count));
}
__device__ __forceinline__ void mbarExpectTx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbarArrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smemAddr(bar)) : "memory");
}
// One poll of a phase.  The suspend-time hint lets the hardware park the thread until the phase
// completes (or the hint runs out) instead of returning at once: a block here has a dozen warps
// waiting for one another most of the time, and warps that spin through an unhinted try_wait
// take the issue slots of the few warps that have work (measured on the int8 decode kernel).
__device__ __forceinline__ bool mbarTryWait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smemAddr(bar)), "r"(parity), "r"(kMbarSuspendNs)
            : "memory");
    return ok != 0;
}
// Whether a phase is complete, without parking the thread.
__device__ __forceinline__ bool mbarTestWait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smemAddr(bar)), "r"(parity)
            : "memory");
    return ok != 0;
}
__device__ __forceinline__ void fenceBarrierInit() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fenceProxyAsync() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- TMA -----------------------------------------------------------------------
__device__ __forceinline__ void tmaPrefetchDesc(const CUtensorMap *m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 3-D tile load global -> shared, completion counted in bytes on `bar`.  The
// innermost coordinate c0 must be a multiple of 16 bytes of elements.
__device__ __forceinline__ void tmaLoad3D(void *dst, const CUtensorMap *m, uint64_t *bar, int c0, int c1,
                                          int c2) {
    asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smemAddr(dst)),
            "l"(reinterpret_cast<uint64_t>(m)), "r"(smemAddr(bar)), "r"(c0), "r"(c1), "r"(c2)
            : "memory");
}
// L2 eviction policies for streaming data: evict_first for rows that are read once, evict_last for
// rows fetched ahead of their use.
__device__ __forceinline__ uint64_t l2PolicyEvictFirst() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ uint64_t l2PolicyEvictLast() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void tmaLoad3DHint(void *dst, const CUtensorMap *m, uint64_t *bar, int c0, int c1, int c2,
                                              uint64_t policy) {
    asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
            " [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(smemAddr(dst)),
            "l"(reinterpret_cast<uint64_t>(m)), "r"(smemAddr(bar)), "r"(c0), "r"(c1), "r"(c2), "l"(policy)
            : "memory");
}
__device__ __forceinline__ void tmaPrefetchL2_3DHint(const CUtensorMap *m, int c0, int c1, int c2, uint64_t policy) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile.L2::cache_hint [%0, {%1, %2, %3}], %4;" ::"l"(
                         reinterpret_cast<uint64_t>(m)),
                 "r"(c0), "r"(c1), "r"(c2), "l"(policy)
                 : "memory");
}
// The same tile pulled into L2 only (no shared-memory destination, no completion to wait for).
__device__ __forceinline__ void tmaPrefetchL2_3D(const CUtensorMap *m, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                         reinterpret_cast<uint64_t>(m)),
                 "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void tmaLoad2D(void *dst, const CUtensorMap *m, uint64_t *bar, int c0, int c1) {
    asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4}], [%2];" ::"r"(smemAddr(dst)),
            "l"(reinterpret_cast<uint64_t>(m)), "r"(smemAddr(bar)), "r"(c0), "r"(c1)
            : "memory");
}
__device__ __forceinline__ void tmaLoad4D(void *dst, const CUtensorMap *m, uint64_t *bar, int c0, int c1,
                                          int c2, int c3) {
    asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smemAddr(dst)),
            "l"(reinterpret_cast<uint64_t>(m)), "r"(smemAddr(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
            : "memory");
}

// ---- cp.async (4-byte, for the scale columns riding in the same stage) -------------
__device__ __forceinline__ void cpAsync4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smemAddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncMbarArriveNoinc(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smemAddr(bar)) : "memory");
}

// ---- warp-level matrix helpers -----------------------------------------------------
__device__ __forceinline__ void ldmatrixX4(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3,
                                           uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldmatrixX4Trans(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3,
                                                uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ uint32_t movmatrixTrans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
// D(16x8,f32) += A(16x16,f16,row) * B(16x8,f16,col)
__device__ __forceinline__ void mmaF16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b0, uint32_t b1) {
    asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D(16x8,f32) += A(16x8,tf32,row) * B(8x8,tf32,col)
__device__ __forceinline__ void mmaTf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
    asm volatile(
            "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t toTf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// ---- exact int8 -> fp16 ----------------------------------------------------------
// A byte u placed in the low mantissa bits of an fp16 with zero exponent IS the
// subnormal u * 2^-24, exactly.  With u = x + 128 (w holds four int8 already xor-ed with
// 0x80) the operand carries a +128 offset that the caller removes after the MMA with a
// per-column sum; one prmt per pair.
template <uint32_t SEL>
__device__ __forceinline__ uint32_t subnormalPair(uint32_t w) {
    return __byte_perm(w, 0u, SEL);
}

// Programmatic dependent launch: wait for the grids this one depends on (and for
// their memory to be visible) / let the dependent grid start its prologue.
__device__ __forceinline__ void gridDepWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void gridDepLaunch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ uint32_t packHalf2(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
}
// x = hi + lo with both parts fp16: the pair carries ~22 mantissa bits.
__device__ __forceinline__ void splitHalf(float x, float &hi, float &lo) {
    hi = __half2float(__float2half_rn(x));
    lo = x - hi;
}

__device__ __forceinline__ float fastExp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void namedBarSync(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void namedBarArrive(uint32_t id, uint32_t threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

#endif  // __CUDACC__

}  // namespace tc
