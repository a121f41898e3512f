// The two-wave search on the device (dummest-search.hh:119-193): the float
// filter (findSimilaritiesBackwardOnly) over every pair, then the full
// mid-anchored scoring over the survivors, with no host round trip.
//
// A pair survives when its float best b is positive and passes the E-value
// gate K_filter T / exp(lambda_filter ln b) <= E_filter, or when b is +inf
// ("inf always survives", dummest-search.hh:163-168).  The gate decreases in b,
// so the host turns it into the smallest float b* that passes
// (dmst_filter_threshold, evaluated with the reference's expression in
// double), and the device compares b >= b*.
//
// The survivors of each chunk of the filter wave (pairs of one profile,
// longest read first) become the pairs of the same chunk of the second wave,
// in order, so the compaction needs no scan across chunks: one warp per chunk
// packs its survivors with a ballot.  They also go to one list, roughly
// costliest first: up to kWaveMax of them run on the stripe pipeline instead,
// one pair after another on each CTA.  Few survivors leave each chunk two or
// three pairs for its 12 warps and a barrier after them: 1,741 of 32,000 pairs
// (M 50-800, reads of 150-3000 nt) took 13 ms as chunks.
#pragma once

#include "dp_common.cuh"
#include "dp_wavefront.cuh"

namespace dmst {

// Survivors that the second wave takes one by one; beyond, the chunks are
// full enough (measured on random pairs of M = 800, L = 3000: the pipeline is
// within 5% of the batched kernel at 4,000 pairs).
constexpr int kWaveMax = 8192;

// count[0]: survivors, in list (device scratch, zeroed).
__global__ void survivorKernel(const Chunk *filterChunks, int nChunks, const PairOut *fo, const float *minBest,
                               Chunk *midChunks, int *survivorIdx, int chunkStride, uint8_t *survived, int *list,
                               int *count) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (c >= nChunks) return;  // whole warps
    const Chunk ch = filterChunks[c];
    const float gate = minBest[ch.prof];
    int cnt = 0;
    for (int k0 = 0; k0 < ch.count; k0 += kLanes) {
        const int k = k0 + lane;
        bool sv = false;
        int pi = 0;
        if (k < ch.count) {
            pi = ch.first + k;
            const float b = fo[pi].filt;
            sv = b > 0.0f && (b >= gate || isinf(b));
            survived[pi] = sv ? 1 : 0;
        }
        const unsigned m = __ballot_sync(kFull, sv);
        if (sv) survivorIdx[(size_t)c * chunkStride + cnt + __popc(m & ((1u << lane) - 1u))] = pi;
        cnt += __popc(m);
    }
    int at = 0;
    if (lane == 0) {
        midChunks[c] = Chunk{c * chunkStride, cnt, ch.prof, ch.rowPad};
        at = cnt ? atomicAdd(count, cnt) : 0;
    }
    at = __shfl_sync(kFull, at, 0);
    __syncwarp();
    for (int k = lane; k < cnt; k += kLanes) list[at + k] = survivorIdx[(size_t)c * chunkStride + k];
}

// Up to kWaveMax survivors run from the list (count[1] of them), and the
// chunks are emptied; more run as chunks (count[1] = 0).
__global__ void wavePlanKernel(Chunk *midChunks, int nChunks, int *count) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const bool listed = count[0] <= kWaveMax;
    if (c == 0) count[1] = listed ? count[0] : 0;
    if (listed && c < nChunks) midChunks[c].count = 0;
}

// The survivors of a small call, whose filter wave ran on the stripe pipeline
// over `all` (costliest first): one thread per pair, count[1] of them in list.
__global__ void survivorListKernel(const int *all, int n, const DevPair *pairs, const PairOut *fo, const float *minBest,
                                   uint8_t *survived, int *list, int *count) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int pi = all[k];
    const float b = fo[pi].filt;
    const bool sv = b > 0.0f && (b >= minBest[pairs[pi].prof] || isinf(b));
    survived[pi] = sv ? 1 : 0;
    if (sv) list[atomicAdd(count + 1, 1)] = pi;
}

}  // namespace dmst
