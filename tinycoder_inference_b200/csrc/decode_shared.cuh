// decode_shared.cuh -- pieces shared by the split-KV decode kernels (int8 store and
// f32/fp16 cache): the bounded mbarrier wait, the chunk plan, the merge launcher.
#pragma once

#include "tc_common.cuh"

namespace tc {

// What a block of n takes of len tokens, in whole 16-token tiles (the decode kernels whose blocks share a device length,
// and the merge behind them).
__host__ __device__ inline uint32_t tokensPerBlock(uint32_t len, uint32_t n) {
    return (((len + 15u) >> 4) + n - 1u) / n * 16u;
}

// q of one token rotated in place by the merge (decode launches whose blocks all still read it leave that to it):
// table row = the token's position = attended rows - 1, at most maxLen - 1.
struct QRotation {
    float *q;                  // nullable: [nHeads][hd]
    const float *cosT, *sinT;  // [rows][hd / 2]
    uint32_t maxLen;
};

// devLens (nullable): the merge works out on the device how many of the activeHost partials were written, from the
// length devLens[s] + lenAdd and chunkTokens per partial (0: tokensPerBlock of the length, at most rot.maxLen).
// early: the grid behind the merge may start while the one that writes the partials still runs.  For an int8 decode at
// head_dim 128 that is the caller's word (TC_DECODE_PDL); the others write no row that any launch reads ahead of its
// wait, and are past their own wait before the merge can start.
int launchMerge(const float *pAcc, const float *pM, const float *pL, float *out, uint32_t seqLen,
                uint32_t nHeads, uint32_t numChunks, uint32_t activeHost, uint32_t hd, const uint32_t *devLens,
                uint32_t lenAdd, uint32_t chunkTokens, uint8_t *q81, bool early, cudaStream_t st,
                uint32_t chunksPerRank = 0, uint64_t rankStride = 0, QRotation rot = {nullptr, nullptr, nullptr, 0});

// An f32 store kept beside an int8 pool: where the appended row of a decode call also goes, verbatim (one
// sequence; row = its last).
struct F32Mirror {
    float *k, *v;  // nullable: [rows][nKV][hd]
};

// `bytes` of K and of V zeroed in stream order, wherever they lie (kv_write.cu)
int kvClear(void *k, void *v, size_t bytes, cudaStream_t st);

// int8 decode (decode_i8.cu): tc_attn_decode_i8_batch plus the mirror; lens[b] + lenAdd is the length on the device
int decodeI8Common(const tc_decode_i8_batch *d, uint32_t lenHost, uint32_t lenAdd, const F32Mirror &mir, cudaStream_t st);
// one sequence whose length the launch need not know (captured decode steps): no partials, one launch
int decodeI8Streams(const tc_decode_i8_batch *d, uint32_t lenHost, uint32_t lenAdd, cudaStream_t st);
// its head_dim 128 form on tcgen05 (decode_i8_tc.cu); arguments already validated
int decodeI8Tc(const tc_decode_i8_batch *d, uint32_t lenHost, uint32_t lenAdd, const F32Mirror &mir, cudaStream_t st);

#ifdef __CUDACC__
// Bounded wait: the first poll, which most waits need alone, in front of a loop of up to 2^18 more, each parked for up to
// 20 us by the hardware.  (A loop that reads the clock: captured int8 step of 28 / 4 / 128 at 12000 rows 23.0 -> 23.6 us per layer,
// 8 sequences of 4098 rows 9.83 -> 9.95.)  TEST: a first poll that does not park.  It is the better one where the phase is nearly
// always complete (tcgen05 decode, 98 calls of 1 - 64 sequences of 16 - 32767 rows: 0.7 % on average, up to 3 % of short ones, where
// two runs differ by 0.1 %) and the worse one where warps do wait (captured step, 5000 rows, 11.95 -> 12.05).
template <bool TEST = false>
__device__ __forceinline__ bool mbarWait(uint64_t *bar, uint32_t parity, unsigned int *err, uint32_t errBit) {
    if (TEST ? mbarTestWait(bar, parity) : mbarTryWait(bar, parity)) return true;
#pragma unroll 1
    for (uint32_t i = 0; i < (1u << 18); ++i)
        if (mbarTryWait(bar, parity)) return true;
    atomicOr(err, errBit);
    return false;
}

#endif

// rowsPerStage = (token, kv-head) rows one pipeline stage holds; a CTA streams
// hpc kv heads, so a stage covers rowsPerStage / hpc tokens.
struct DecodePlan {
    uint32_t hpc, headGroups, chunkTokens, chunksPerSeq, tileTokens;
};

// One wave of CTAs over the SMs when every sequence has the same (host-known) length: a second
// wave only adds a tail (measured, 8 sequences of 32768 rows: 48.5 us per layer with one wave,
// 53.3 with two, 56.7 with three).  Lengths that live on the device may be ragged: chunks are cut
// by the longest sequence, short sequences leave most of theirs empty, and four waves of small
// chunks let the hardware scheduler even things out (64 sequences in [512, 32768]: 182 us with
// four waves, 186 with two, 324 with one).
inline DecodePlan planDecode(uint32_t batch, uint32_t nKV, uint32_t maxLen, uint32_t slots, uint32_t rowsPerStage,
                             bool uniformLengths = true, uint32_t maxHpc = 4) {
    DecodePlan pl;
    pl.hpc = (nKV % 4u == 0 && maxHpc >= 4u) ? 4u : ((nKV % 2u == 0 && maxHpc >= 2u) ? 2u : 1u);
    pl.headGroups = nKV / pl.hpc;
    pl.tileTokens = rowsPerStage / pl.hpc;
    const uint32_t tilesMax = (maxLen + pl.tileTokens - 1) / pl.tileTokens;
    const uint32_t sms = static_cast<uint32_t>(numSMs());
    // (four waves of blocks that stream four kv heads each; a block that streams fewer kv heads gets
    // proportionally more of them, so that a block covers the same token range: 64 ragged sequences
    // with one kv head per block: 204 us at 4 waves, 184 at 8 and 16, 206 at 32)
    const uint32_t waves = (batch > 1 && !uniformLengths) ? 4u * (4u / pl.hpc) : 1u;
    uint32_t want = (sms * waves) / (batch * pl.headGroups);
    want = want < 1u ? 1u : want;
    // ragged batches: never cut a sequence finer than about 24 stages per block -- with few sequences per
    // GPU the wave rule alone leaves blocks of a few tiles whose set-up costs more than their work
    if (waves > 1u && want > (tilesMax + 23u) / 24u) want = (tilesMax + 23u) / 24u;
    want = want > slots ? slots : want;
    want = want > tilesMax ? tilesMax : want;
    want = want < 1u ? 1u : want;
    const uint32_t tilesPerChunk = (tilesMax + want - 1) / want;
    pl.chunkTokens = tilesPerChunk * pl.tileTokens;
    pl.chunksPerSeq = (tilesMax + tilesPerChunk - 1) / tilesPerChunk;
    if (pl.chunksPerSeq == 0) pl.chunksPerSeq = 1;
    return pl;
}


}  // namespace tc
