// prefill_rows.cuh -- the tensor-core prefill as the session calls it (prefill_f16.cu): the store the rows live in,
// the rows a call brings, the int8 pool beside an f32 store.
#pragma once

#include "tc_common.cuh"

namespace tc {

// Where the int8 mirror of the call's new K/V rows goes (the reference keeps such a pool beside its
// f32 store and rebuilds it before the first decode step, GPUComputeMoE.cu:3049-3063): rows
// [cachePos, cachePos + seqLen) of the cache become pool rows dstRow ..; null k8 = no mirror.
struct PrefillMirror {
    int8_t *k8, *v8;   // [rows][nKV][hd]
    float *ks, *vs;    // [rows][nKV]
    uint64_t dstRow;   // pool row of cache row cachePos
    uint64_t maxRows;  // rows the pool holds
};

// The store of a call's K/V rows: f32 (twins made), fp16 (used in place: its layout is the twins'), or int8 (twins made:
// byte x the row's scale).  Written only for rows the call brings.
struct PrefillKvStore {
    int kind;        // 0 f32, 1 fp16, 2 int8
    void *k, *v;     // [rows][nKV][hd] of float / __half / int8_t
    float *ks, *vs;  // int8: [rows][nKV] scales
};

// The K/V rows of a call that are not in the store yet (null k: they are): f32 [seqLen][nKV][hd], stored at rows
// cachePos ..; with tables [rows][hd / 2] K, and q in place, are rotated by table row = cache row first.
struct PrefillNewRows {
    const float *k, *v;
    const float *cosT, *sinT;
};

int prefillF16(float *q, const PrefillKvStore &src, float *out, void *scratch, size_t scratchBytes, uint32_t seqLen,
               uint32_t cachePos, uint32_t nHeads, uint32_t nKV, uint32_t hd, float invSqrt, const PrefillMirror &mir,
               const PrefillNewRows &nr, cudaStream_t st);

}  // namespace tc
