// Exact row-rescaled DP for the pairs the fast kernels cannot score exactly (a
// row maximum above RESCALE_THRESH, or a product beyond float range): one pair
// on all warps of a CTA, or of a cluster of CTAs.
//
// The reference decides each row's rescale after the whole row is known
// (dummest-dp-backward.hh:560-573, dummest-dp-forward.hh:228-242), which a
// wavefront cannot wait for.  So each direction runs twice (the kDiscover
// and kReplay modes of the step functions below):
//
//  1. discovery: the same recurrence with a per-lane scale count that rises
//     by one (values x 2^-64, exact) whenever a value passes 2^100, and that
//     lanes align when they exchange values.  Every operation then sees the
//     reference's operands up to an exact power of two, so each row's
//     maximum is the reference's up to that power; the row's (max, count)
//     is recorded.  A scan over the rows turns these into the reference's
//     own counts: cnt_i = cnt_prev + [max_i * 2^(64 (count_i - cnt_prev)) > 1e30].
//  2. replay: the reference's arithmetic exactly, with those counts known in
//     advance: row i computes at the scale of the row it reads, seeds times
//     2^(-64 cnt_prev), and multiplies everything it hands on (stored W1, the
//     values sent to the next row) by 2^-64 when its own count rose.
//
// Mid and filter maxima are taken over exact double products (the reference
// forms them in double and rounds the mantissa to float,
// dummest-batch.hh:146-235) and folded with the row's count sum into an
// exact (mantissa, exponent) best.
//
// Schedule.  Profile stripe s (32 R rows) runs on warp s mod G of the cluster
// in every sweep, so that a lane reads back the W1 it stored.  Boundary rows
// pass through one 16-byte ring entry per column and stripe, each half its own
// flag (dp_pipe.cuh): kRingEmpty until written, emptied again by its reader,
// which loads a block ahead.  Both discovery sweeps follow each other without
// a barrier (neither reads the other's values), or run side by side on twice
// as many warps as stripes; then the counts are scanned, then both replay
// sweeps.  Every wait is for an earlier stripe of the same
// cluster and bounded: a wait that runs out sets the ring buffer's abort flag
// (dp_pipe.cuh), every warp leaves its sweep, and the pair and those started
// after it are marked failed, also by a kernel queued before the host knows.
//
// Bound: the latency of a step, so two rows per lane, one column apart
// (dp_stagger.cuh: neither waits for the other), on as many warps as there are
// stripes; steps inside the read run without masks, and the FP64 products are
// formed only for cells that can raise a row's best (rowBestFold).  Measured:
// three windows of 10 kb against M = 2000 in 8.3 ms (170 ns a step), 10.8 with
// the discovery sweeps in turn, 18.7 with two rows at one column and every
// product, 47 with four rows per lane on the 8 warps of one CTA; 55 pairs of M
// = 400 x 2.2 kb in 1.8, 2.0, 4.0 and 8.5 ms.
#pragma once

#include "dp_exact.cuh"
#include "dp_pipe.cuh"
#include "dp_traceback_job.cuh"

namespace dmst {

constexpr int kExactRows = 2;  // rows per lane
constexpr int kExactStripe = kLanes * kExactRows;
constexpr int kExactMaxWarps = 15;  // 227 KB of windows
// Shared memory of a warp: the fast path's window, the discovery's ring counts
// (mirrored like the ring), and the stripe's emission rows, code-major.
struct WindowX {
    WindowS<kExactRows> s;
    int cnt[kSRingWin + kSBlock];
    float emit[kNumCodes * kExactStripe];
};

__host__ __device__ inline int exactStripes(int M) { return (M + kExactStripe) / kExactStripe; }
// Scratch of a cluster (floats): W1 by stripe and step, row maxima and
// counts of both discovery sweeps, reference counts, the warps' bests, and
// with anchors the stripes' column partials.
__host__ __device__ inline long long exactW1Floats(int M, int L) {
    return exactStripes(M) * pipeStripeFloats(L, kExactRows);
}
__host__ __device__ inline long long exactPipeScratch(int M, int L, bool anchors) {
    const long long rows = 4LL * (M + 1) + 2LL * (M + 2);
    return (exactW1Floats(M, L) + rows + 8LL * kPipeMaxCluster * kExactMaxWarps + 64 +
            (anchors ? 3LL * exactStripes(M) * L : 0) + 63) / 64 * 64;
}
// Ring words (64-bit, two per entry) of a cluster: both directions.
__host__ __device__ inline long long exactRingWords(int M, int L) { return 4LL * exactStripes(M) * L; }

struct ExactPipeArgs {
    const int *queue;       // flagged pairs, costliest first
    const int *queueCount;
    const DevPair *pairs;
    const DevProfile *profiles;
    const float *emit, *params;
    const uint8_t *codes;
    const float *seeds;
    const PairScales *scales;
    float *pool;
    long long poolSlot;     // floats per cluster
    unsigned long long *ring;
    long long ringSlot;     // words per cluster
    int *abort;             // the ring buffer's flag, 0 while every word is empty between kernels
    ExactOut *out;
    // anchors: anchorOff[pair] >= 0 is the offset of its L columns
    const long long *anchorOff;
    float *anchorM;
    int *anchorE, *anchorRow;
    // traceback jobs (jobOf[pair] >= 0): the replay sweeps' W0 and then W1
    // before each row's rescale, by stripe and step (at AlignJob::stepOff in
    // alignSteps; alignRowsKernel makes them row-major) and the reference's
    // rescale counts (AlignJob::rowOff in alignRows: cntB at [0, M+2), cntF
    // after it)
    const int *jobOf;
    const AlignJob *jobs;
    float *alignSteps;
    int *alignRows;
    int spinLimit;          // polls of a wait before it gives up
};

// A block's window entry of a lane, as loaded.
struct FillX {
    FillP p;
    unsigned long long cnt;
};

template <bool BACKWARD, bool DISCOVER>
__device__ __forceinline__ FillX fillLoadX(const SweepArgs &a, const unsigned long long *in, int u) {
    FillX f{fillLoadP<BACKWARD>(a, nullptr, u), 0ull};
    if (in && u < a.L) {
        f.p.ring = ringPeek(in + 2 * (size_t)u);
        if (DISCOVER) f.cnt = ringPeek(in + 2 * (size_t)u + 1);
    }
    return f;
}

// The window entry of local time u, once its ring values are there; false:
// given up.
template <bool BACKWARD, bool DISCOVER>
__device__ __forceinline__ bool fillStoreX(WindowX &w, const SweepArgs &a, FillX f, unsigned long long *in, int u,
                                           int *abort, int spinLimit) {
    if (in) {
        int it = 0;
        auto empty = [&]() { return f.p.ring == kRingEmpty || (DISCOVER && f.cnt == kRingEmpty); };
        while (__any_sync(kFull, empty())) {
            if (empty()) {
                f.p.ring = ringPeek(in + 2 * (size_t)u);
                if (DISCOVER) f.cnt = ringPeek(in + 2 * (size_t)u + 1);
            }
            if (++it > spinLimit || (it & 63) == 0) {
                const bool gone = it > spinLimit || abortPeek(abort) != 0;
                if (__any_sync(kFull, gone)) {
                    *reinterpret_cast<volatile int *>(abort) = 1;
                    return false;
                }
            }
        }
        if (u < a.L) {
            ringPut(in + 2 * (size_t)u, kRingEmpty);
            if (DISCOVER) ringPut(in + 2 * (size_t)u + 1, kRingEmpty);
        }
    }
    const FillRegs r{f.p.code, f.p.suf, f.p.pre, __uint_as_float((unsigned)f.p.ring),
                     __uint_as_float((unsigned)(f.p.ring >> 32))};
    fillStoreS<BACKWARD, kExactRows>(w.s, a, r, u);
    if (DISCOVER) {
        const int e = u & (kSRingWin - 1);
        w.cnt[e] = (int)f.cnt;
        if (e < kSBlock) w.cnt[e + kSRingWin] = (int)f.cnt;
    }
    return true;
}

// Two ring words of a column: (W, Y), and in the discovery its scale count.
template <bool DISCOVER>
__device__ __forceinline__ void ringPutX(unsigned long long *p, float w, float y, int cnt) {
    ringPut(p, ((unsigned long long)__float_as_uint(y) << 32) | __float_as_uint(w));
    if (DISCOVER) ringPut(p + 1, (unsigned)cnt);
}

// The largest exact product of a row, and the sum of its factors' bits as a
// cheap upper test: the bits of a positive float are 2^23 times its binary
// logarithm (biased) less at most 0.0861 2^23, so a product whose bit sum is
// kBitSlack below the best's is smaller, and the double product, the
// comparison and the select are left out for it (most cells).
constexpr unsigned kBitSlack = 1445000;  // 2 x 0.0861 x 2^23, rounded up
struct RowBest {
    double v;
    unsigned floor;
};
__device__ __forceinline__ void rowBestFold(RowBest &b, float x, float y) {
    const unsigned bx = __float_as_uint(x), s = bx + __float_as_uint(y);
    if (s >= b.floor && bx != 0) {
        const double p = (double)x * (double)y;
        if (p > b.v) {
            b.v = p;
            b.floor = s - kBitSlack;
        }
    }
}

// ---------------------------------------------------------------------------
// The staggered steps of the exact path (dp_stagger.cuh's, two rows per lane,
// with the discovery's scale counts or the replay's row factors).  GEN: steps
// at which some lane is outside the read.
// ---------------------------------------------------------------------------
struct RunX {
    const float4 *col;
    const float2 *ring;
    const int *cnt;
    float *w1;
    float *align;
    unsigned long long *out;
};

template <int MODE>
struct BwdX {
    Coef<kExactRows> c;
    float h[4][2], z[4][2], rb[4], yPrev[2];
    float ho[4];  // replay: row 1's W1 history as it leaves the row (after its rescale)
    float bgH[4], sufH[4], preH[4], evH[4][2];
    float sendW, sendY;
    int u;
    float *wp;
    unsigned eS;
    // discovery
    int cnt, sendC;
    float rmax[2];
    // replay
    float fOut[2];
    int cOut[2];
    RowBest best[2];
    float *align;  // this step's W1 before the rows' rescale (traceback), or null
};

// Scales the lane's state by f and takes the count cnt (discovery).
__device__ __forceinline__ void bwdRescaleX(BwdX<kDiscover> &b, float f, int cnt, int row, int M) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            b.h[q][k] *= f;
            b.z[q][k] *= f;
        }
        b.rb[q] *= f;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        b.yPrev[k] *= f;
        b.rmax[k] *= f;
        b.c.rs[k] = seedCoef(row + k <= M, cnt);
    }
    b.cnt = cnt;
}

template <int MODE, int PH, bool GEN>
__device__ __forceinline__ void bwdStepX(BwdX<MODE> &b, const SweepArgs &a, WindowX &w, int lane, int row, int M,
                                         unsigned long long *out, const RunX &ip) {
    constexpr int R = kExactRows;
    constexpr bool kDisc = MODE == kDiscover;
    constexpr int SW = kLanes * R;
    float inW = __shfl_down_sync(kFull, b.sendW, 1);
    float inY = __shfl_down_sync(kFull, b.sendY, 1);
    int inC = 0;
    if (kDisc) inC = __shfl_down_sync(kFull, b.sendC, 1);
    const float4 col = GEN ? w.s.col[b.u & (kSWin - 1)] : ip.col[PH];
    if (lane == kLanes - 1) {
        const float2 r = GEN ? w.s.ring[b.u & (kSRingWin - 1)] : ip.ring[PH];
        inW = r.x;
        inY = r.y;
        if (kDisc) inC = GEN ? w.cnt[b.u & (kSRingWin - 1)] : ip.cnt[PH];
    }
    if constexpr (kDisc) {
        // the incoming values and this lane to one scale
        if ((!GEN || (b.u >= 0 && b.u < a.L + R)) && inC != b.cnt) {
            if (inC > b.cnt) {
                bwdRescaleX(b, stepsDown(inC - b.cnt), inC, row, M);
            } else {
                const float f = stepsDown(b.cnt - inC);
                inW *= f;
                inY *= f;
            }
        }
    }
    float ev[R];
    loadEmitS<R>(ev, b.eS + 4u * (unsigned)__float_as_int(col.x));
    b.bgH[PH] = col.y;
    b.sufH[PH] = col.z;
    b.preH[PH] = col.w;
#pragma unroll
    for (int k = 0; k < R; ++k) b.evH[PH][k] = ev[k];
    b.rb[PH] = inW;
    float nW[R], nY[R], nZ[R], pv[R];
    bool act[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int D = R - 1 - k;
        const int Q = (PH + 4 - D) & 3;
        pv[k] = b.preH[Q];
        float Wb1, Wb2, Wb3, Yb;  // the row below: W1 at columns j+1, j+2, j+3 and Y at j
        if (k == R - 1) {
            Wb1 = b.rb[(PH + 3) & 3];
            Wb2 = b.rb[(PH + 2) & 3];
            Wb3 = b.rb[(PH + 1) & 3];
            Yb = inY;
        } else if (kDisc) {
            Wb1 = b.h[(PH + 2) & 3][k + 1];
            Wb2 = b.h[(PH + 1) & 3][k + 1];
            Wb3 = b.h[PH][k + 1];
            Yb = b.yPrev[k + 1];
        } else {
            Wb1 = b.ho[(PH + 2) & 3];
            Wb2 = b.ho[(PH + 1) & 3];
            Wb3 = b.ho[PH];
            Yb = b.yPrev[k + 1];
        }
        const float p = (Wb3 * b.evH[Q][k]) * b.c.enter[k];
        float acc = __fmaf_rn(Yb, b.c.d0[k], p);
        acc = __fmaf_rn(Wb2, b.c.d1[k], acc);
        acc = __fmaf_rn(Wb1, b.c.d2[k], acc);
        const float zbg = b.z[(PH + 1) & 3][k] * b.bgH[Q];
        acc = __fmaf_rn(zbg, b.c.a0[k], acc);
        acc = __fmaf_rn(b.h[(PH + 2) & 3][k], b.c.a2[k], acc);
        acc = __fmaf_rn(b.h[(PH + 3) & 3][k], b.c.a1[k], acc);
        float W = __fmaf_rn(b.sufH[Q], b.c.rs[k], acc);
        float Y = __fmaf_rn(b.c.eps[k], Yb, W);
        float Z = __fmaf_rn(b.c.b0[k], zbg, W);
        act[k] = true;
        if (GEN) {
            act[k] = b.u >= D && b.u < a.L + D;
            if (!act[k]) W = Y = Z = 0.0f;
        }
        nW[k] = W;
        nY[k] = Y;
        nZ[k] = Z;
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        b.h[PH][k] = nW[k];
        b.z[PH][k] = nZ[k];
        if (kDisc) {
            b.rmax[k] = fmaxf(b.rmax[k], nY[k]);  // Y >= W1 at every cell
            b.yPrev[k] = nY[k];
        }
    }
    if constexpr (kDisc) {
        if (fmaxf(nY[0], nY[1]) > kBump) bwdRescaleX(b, kStep, b.cnt + 1, row, M);
        b.sendW = b.h[PH][0];
        b.sendY = b.yPrev[0];
        b.sendC = b.cnt;
    } else {
        if (b.align != nullptr) storeW1S<R>(GEN ? b.align : ip.align + PH * SW, nW);
        // what leaves a row is scaled by the row's own decision
        float oW[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            oW[k] = nW[k] * b.fOut[k];
            b.yPrev[k] = nY[k] * b.fOut[k];
            rowBestFold(b.best[k], oW[k], pv[k]);
        }
        b.ho[PH] = oW[1];
        b.sendW = oW[0];
        b.sendY = b.yPrev[0];
        storeW1S<R>(GEN ? b.wp : ip.w1 + PH * SW, oW);
    }
    if (lane == 0 && out != nullptr) {
        if (GEN) {
            if (act[0]) ringPutX<kDisc>(out + 2 * (ptrdiff_t)(b.u - (R - 1)), b.sendW, b.sendY, b.cnt);
        } else {
            ringPutX<kDisc>(ip.out + 2 * PH, b.sendW, b.sendY, b.cnt);
        }
    }
    if (GEN) {  // otherwise the run advances them
        b.wp += SW;
        if (!kDisc && b.align != nullptr) b.align += SW;
        ++b.u;
    }
}

// One stripe of a backward sweep; `out`: its ring to the stripe below.
template <int MODE>
__device__ bool exactBackward(const SweepArgs &a, WindowX &w, int s, int lane, unsigned long long *in,
                              unsigned long long *out, int *abort, int spinLimit, const ExactRows &x,
                              ExactBest *exact) {
    constexpr int R = kExactRows, S = kExactStripe, SW = kLanes * R;
    constexpr bool kDisc = MODE == kDiscover;
    const int M = a.M(), row = s * S + lane * R;
    BwdX<MODE> b;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < R; ++k) b.h[q][k] = b.z[q][k] = b.evH[q][k] = 0.0f;
        b.rb[q] = b.ho[q] = b.bgH[q] = b.sufH[q] = b.preH[q] = 0.0f;
    }
    loadBackwardCoef<R>(b.c, a, row);
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int i = row + k;
        b.yPrev[k] = b.rmax[k] = 0.0f;
        b.best[k] = RowBest{0.0, 0u};
        b.fOut[k] = 1.0f;
        b.cOut[k] = 0;
        if (!kDisc) {
            const int ci = i <= M ? i : M + 1;
            const int cIn = __ldcg(x.cntB + min(ci + 1, M + 1));
            b.cOut[k] = __ldcg(x.cntB + ci);
            b.fOut[k] = stepsDown(b.cOut[k] - cIn);
            b.c.rs[k] = seedCoef(i <= M, cIn);
        }
    }
    b.sendW = b.sendY = 0.0f;
    b.cnt = b.sendC = 0;
    b.u = -(kLanes - 1 - lane) * R;
    b.wp = a.w1 + lane * R;
    b.eS = (unsigned)__cvta_generic_to_shared(a.smE + lane * R);
    b.align = !kDisc && a.alignOut ? a.alignOut + lane * R : nullptr;
    const int T = (a.L - 1 + S + 3) / 4 * 4;
    for (int v = -S + lane; v < 0; v += kLanes) fillStoreX<true, kDisc>(w, a, FillX{{kPad, 0.0f, 0.0f, 0ull}, 0ull}, nullptr, v, abort, 0);
    __syncwarp();
    FillX f = fillLoadX<true, kDisc>(a, in, lane);
    if (!fillStoreX<true, kDisc>(w, a, f, in, lane, abort, spinLimit)) return false;
    f = fillLoadX<true, kDisc>(a, in, kSBlock + lane);
    for (int t0 = 0; t0 < T; t0 += kSBlock) {
        __syncwarp();
        if (!fillStoreX<true, kDisc>(w, a, f, in, t0 + kSBlock + lane, abort, spinLimit)) return false;
        f = fillLoadX<true, kDisc>(a, in, t0 + 2 * kSBlock + lane);
        __syncwarp();
        const int n = min(kSBlock, T - t0);
        int gA, gB;
        interiorRunS<4>(a, S, t0, n, gA, gB);
        int g = 0;
        RunX ip{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
#pragma unroll 1
        for (; g < gA; g += 4) {
            bwdStepX<MODE, 0, true>(b, a, w, lane, row, M, out, ip);
            bwdStepX<MODE, 1, true>(b, a, w, lane, row, M, out, ip);
            bwdStepX<MODE, 2, true>(b, a, w, lane, row, M, out, ip);
            bwdStepX<MODE, 3, true>(b, a, w, lane, row, M, out, ip);
        }
        if (gB > gA) {
            ip.col = w.s.col + (b.u & (kSWin - 1));
            ip.ring = w.s.ring + (b.u & (kSRingWin - 1));
            ip.cnt = w.cnt + (b.u & (kSRingWin - 1));
            ip.w1 = b.wp;
            ip.align = b.align;
            ip.out = out + 2 * (ptrdiff_t)(b.u - (R - 1));
#pragma unroll 1
            for (; g < gB; g += 4) {
                bwdStepX<MODE, 0, false>(b, a, w, lane, row, M, out, ip);
                bwdStepX<MODE, 1, false>(b, a, w, lane, row, M, out, ip);
                bwdStepX<MODE, 2, false>(b, a, w, lane, row, M, out, ip);
                bwdStepX<MODE, 3, false>(b, a, w, lane, row, M, out, ip);
                ip.col += 4;
                ip.ring += 4;
                ip.cnt += 4;
                ip.w1 += 4 * SW;
                ip.align += 4 * SW;
                ip.out += 8;
            }
            b.u += gB - gA;
            b.wp += (gB - gA) * SW;
            if (b.align != nullptr) b.align += (gB - gA) * SW;
        }
#pragma unroll 1
        for (; g < n; g += 4) {
            bwdStepX<MODE, 0, true>(b, a, w, lane, row, M, out, ip);
            bwdStepX<MODE, 1, true>(b, a, w, lane, row, M, out, ip);
            bwdStepX<MODE, 2, true>(b, a, w, lane, row, M, out, ip);
            bwdStepX<MODE, 3, true>(b, a, w, lane, row, M, out, ip);
        }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if (row + k > M) continue;
        if (kDisc) {
            x.rowMax[row + k] = b.rmax[k];
            x.rowCnt[row + k] = b.cnt;
        } else {
            foldBest(*exact, b.best[k].v, b.cOut[k]);
        }
    }
    return true;
}

// A column's best wMid on its way up the rows, and its row.
struct Anchor {
    float m;
    int e, row;
};

template <int MODE>
struct FwdX {
    Coef<kExactRows> c;
    float w[4][2], z[4][2], ninPrev[2], yPrev[2];
    float bgH[4], preH[4], evH[4][2];
    float sendIn, sendY;
    int u;
    unsigned eS;
    const float *w1src;
    int gAhead;
    // discovery
    int cnt, sendC;
    float rmax[2];
    // replay
    float fOut[2];
    int cSum[2];  // the row's forward count (before the row) plus its backward count
    RowBest best[2];
    Anchor an[2];  // anchors: per row, the column's best up to it
    float *align;  // this step's W0 (traceback), or null
};

__device__ __forceinline__ void fwdRescaleX(FwdX<kDiscover> &f, float g, int cnt, int row, int M) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            f.w[q][k] *= g;
            f.z[q][k] *= g;
        }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        f.ninPrev[k] *= g;
        f.yPrev[k] *= g;
        f.rmax[k] *= g;
        f.c.rs[k] = seedCoef(row + k <= M, cnt);
    }
    f.cnt = cnt;
}

template <int MODE, int PH, bool GEN, bool ANCH>
__device__ __forceinline__ void fwdStepX(FwdX<MODE> &f, const SweepArgs &a, WindowX &w, int s, int lane, int row, int M,
                                         unsigned long long *out, float *part, const RunX &ip) {
    constexpr int R = kExactRows;
    constexpr bool kDisc = MODE == kDiscover;
    constexpr int SW = kLanes * R;
    constexpr int H = PH & 3;
    float q[R] = {0.0f, 0.0f};
    if (!kDisc) {
        cpAsyncWait<kSW1Ahead - 1>();
        const float2 v = *reinterpret_cast<const float2 *>(&w.s.w1[PH][lane * 2]);
        q[0] = v.x;
        q[1] = v.y;
    }
    float inW = __shfl_up_sync(kFull, f.sendIn, 1);
    float inY = __shfl_up_sync(kFull, f.sendY, 1);
    int inC = 0;
    if (kDisc) inC = __shfl_up_sync(kFull, f.sendC, 1);
    Anchor inA{0.0f, 0, 0};
    if (ANCH) {
        inA.m = __shfl_up_sync(kFull, f.an[R - 1].m, 1);
        inA.e = __shfl_up_sync(kFull, f.an[R - 1].e, 1);
        inA.row = __shfl_up_sync(kFull, f.an[R - 1].row, 1);
        if (lane == 0) inA = Anchor{0.0f, 0, 0};  // the rows below are another stripe's partial
    }
    const float4 col = GEN ? w.s.col[f.u & (kSWin - 1)] : ip.col[PH];
    if (lane == 0) {
        const float2 r = GEN ? w.s.ring[f.u & (kSRingWin - 1)] : ip.ring[PH];
        inW = r.x;
        inY = r.y;
        if (kDisc) inC = GEN ? w.cnt[f.u & (kSRingWin - 1)] : ip.cnt[PH];
    }
    if constexpr (kDisc) {
        if ((!GEN || (f.u >= 0 && f.u < a.L + R)) && inC != f.cnt) {
            if (inC > f.cnt) {
                fwdRescaleX(f, stepsDown(inC - f.cnt), inC, row, M);
            } else {
                const float g = stepsDown(f.cnt - inC);
                inW *= g;
                inY *= g;
            }
        }
    }
    float ev[R];
    loadEmitS<R>(ev, f.eS + 4u * (unsigned)__float_as_int(col.x));
    f.bgH[H] = col.y;
    f.preH[H] = col.z;
#pragma unroll
    for (int k = 0; k < R; ++k) f.evH[H][k] = ev[k];
    float nW[R], nZ[R], nN[R], nY[R];
    bool act[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int Q = (H + 4 - k) & 3;
        const float win0 = k == 0 ? inW : f.ninPrev[k - 1];
        const float yab = k == 0 ? inY : f.yPrev[k - 1];
        const float w1 = f.w[(H + 3) & 3][k], w2 = f.w[(H + 2) & 3][k], w3 = f.w[(H + 1) & 3][k];
        const float X = (f.c.enter[k] * f.evH[Q][k]) * w3;
        float Z0 = f.bgH[Q] * __fmaf_rn(f.c.b0[k], f.z[(H + 1) & 3][k], f.c.a0[k] * w3);
        const float zs = __fmaf_rn(f.c.a2[k], w2, __fmaf_rn(f.c.a1[k], w1, Z0));
        float W0 = win0 + __fmaf_rn(f.preH[Q], f.c.rs[k], zs);
        float Y0 = __fmaf_rn(f.c.eps[k], yab, f.c.d0[k] * W0);
        float nin = __fmaf_rn(f.c.d2[k], w1, __fmaf_rn(f.c.d1[k], w2, X + Y0));
        act[k] = true;
        if (GEN) {
            act[k] = f.u >= k && f.u < a.L + k;
            if (!act[k]) W0 = Y0 = nin = Z0 = 0.0f;
        }
        nW[k] = W0;
        nZ[k] = Z0;
        nN[k] = nin;
        nY[k] = Y0;
    }
    if constexpr (!kDisc) {
        if (ANCH) {
            // wMid = promote(W0) promote(W1): the exact double product, its
            // mantissa rounded to float (dummest-batch.hh:216-235); rows in
            // ascending order, the first row on ties (row k folds what row
            // k - 1 left for its column a step ago)
            const Anchor from[R] = {inA, f.an[0]};
#pragma unroll
            for (int k = 0; k < R; ++k) {
                Anchor an = from[k];
                const unsigned bw = __float_as_uint(nW[k]), bq = __float_as_uint(q[k]);
                if (act[k] && row + k <= M && bw != 0 && bq != 0 &&
                    (an.m == 0.0f || (int)(bw >> 23) + (int)(bq >> 23) - 252 + kRescaleBits * f.cSum[k] >= an.e)) {
                    // the double product's split, from the float mantissas (null_model.cuh):
                    // the replay of 55 hits of M = 400 x 2.2 kb takes 2.9 ms, 3.3 in double
                    const XS v = mulF(XS{__uint_as_float((bw & 0x7FFFFFu) | 0x3F000000u), (int)(bw >> 23) - 126},
                                      XS{__uint_as_float((bq & 0x7FFFFFu) | 0x3F000000u),
                                         (int)(bq >> 23) - 126 + kRescaleBits * f.cSum[k]});
                    if (xsLessMe(an.m, an.e, v.m, v.e)) an = Anchor{v.m, v.e, row + k};
                }
                f.an[k] = an;
            }
            if (lane == kLanes - 1 && act[R - 1]) {
                float *pp = part + ((size_t)s * a.L + (f.u - (R - 1))) * 3;
                pp[0] = f.an[R - 1].m;
                pp[1] = __int_as_float(f.an[R - 1].e);
                pp[2] = __int_as_float(f.an[R - 1].row);
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k) rowBestFold(f.best[k], nW[k], q[k]);
        if (f.align != nullptr) storeW1S<R>(GEN ? f.align : ip.align + PH * SW, nW);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        f.w[H][k] = nW[k];
        f.z[H][k] = nZ[k];
        f.ninPrev[k] = kDisc ? nN[k] : nN[k] * f.fOut[k];
        f.yPrev[k] = kDisc ? nY[k] : nY[k] * f.fOut[k];
        if (kDisc) f.rmax[k] = fmaxf(f.rmax[k], fmaxf(nW[k], nY[k]));
    }
    if constexpr (kDisc) {
        if (fmaxf(fmaxf(fmaxf(nW[0], nY[0]), fmaxf(nW[1], nY[1])), fmaxf(nN[0], nN[1])) > kBump)
            fwdRescaleX(f, kStep, f.cnt + 1, row, M);
        f.sendC = f.cnt;
    }
    f.sendIn = f.ninPrev[R - 1];
    f.sendY = f.yPrev[R - 1];
    if (lane == kLanes - 1 && out != nullptr) {
        if (GEN) {
            if (act[R - 1]) ringPutX<kDisc>(out + 2 * (ptrdiff_t)(f.u - (R - 1)), f.sendIn, f.sendY, f.cnt);
        } else {
            ringPutX<kDisc>(ip.out + 2 * PH, f.sendIn, f.sendY, f.cnt);
        }
    }
    if (!kDisc) {
        float *slot = &w.s.w1[(PH + kSW1Ahead) % kSW1Slots][lane * R];
        if (GEN) {
            if (f.gAhead >= 0) cpAsyncStage<R>(slot, f.w1src);
        } else {
            cpAsyncStage<R>(slot, ip.w1 - PH * SW);
        }
        cpAsyncCommit();
    }
    if (GEN) {
        f.w1src -= SW;
        --f.gAhead;
        if (!kDisc && f.align != nullptr) f.align += SW;
        ++f.u;
    } else if (ANCH) {
        ++f.u;  // otherwise the run advances it
    }
}

// One stripe of a forward sweep; part: the columns' partial anchors (ANCH).
template <int MODE, bool ANCH>
__device__ bool exactForward(const SweepArgs &a, WindowX &w, int s, int lane, unsigned long long *in,
                             unsigned long long *out, int *abort, int spinLimit, const ExactRows &x, ExactBest *exact) {
    constexpr int R = kExactRows, S = kExactStripe, SW = kLanes * R;
    constexpr bool kDisc = MODE == kDiscover;
    const int M = a.M(), row = s * S + lane * R;
    FwdX<MODE> f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < R; ++k) f.w[q][k] = f.z[q][k] = f.evH[q][k] = 0.0f;
        f.bgH[q] = f.preH[q] = 0.0f;
    }
    loadForwardCoef<R>(f.c, a, row);
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int i = row + k;
        f.ninPrev[k] = f.yPrev[k] = f.rmax[k] = 0.0f;
        f.best[k] = RowBest{0.0, 0u};
        f.an[k] = Anchor{0.0f, 0, 0};
        f.fOut[k] = 1.0f;
        f.cSum[k] = 0;
        if (!kDisc) {
            const int ci = i <= M ? i : M;
            const int cIn = __ldcg(x.cntF + ci);
            f.fOut[k] = stepsDown(__ldcg(x.cntF + ci + 1) - cIn);
            f.cSum[k] = cIn + __ldcg(x.cntB + ci);
            f.c.rs[k] = seedCoef(i <= M, cIn);
        }
    }
    f.sendIn = f.sendY = 0.0f;
    f.cnt = f.sendC = 0;
    f.u = -lane * R;
    f.eS = (unsigned)__cvta_generic_to_shared(a.smE + lane * R);
    f.align = !kDisc && a.alignOut ? a.alignOut + lane * R : nullptr;
    const int steps = a.L - 1 + S;
    const int T = (steps + kSW1Slots - 1) / kSW1Slots * kSW1Slots;
    f.w1src = a.w1 + (size_t)(steps - 1) * SW + lane * R;
    f.gAhead = steps - 1 - kSW1Ahead;
    if (!kDisc) {
#pragma unroll
        for (int k = 0; k < kSW1Ahead; ++k) {
            cpAsyncStage<R>(&w.s.w1[k][lane * R], f.w1src);
            cpAsyncCommit();
            f.w1src -= SW;
        }
    }
    for (int v = -S + lane; v < 0; v += kLanes) fillStoreX<false, kDisc>(w, a, FillX{{kPad, 0.0f, 0.0f, 0ull}, 0ull}, nullptr, v, abort, 0);
    __syncwarp();
    FillX p = fillLoadX<false, kDisc>(a, in, lane);
    bool ok = fillStoreX<false, kDisc>(w, a, p, in, lane, abort, spinLimit);
    if (ok) p = fillLoadX<false, kDisc>(a, in, kSBlock + lane);
    for (int t0 = 0; ok && t0 < T; t0 += kSBlock) {
        __syncwarp();
        ok = fillStoreX<false, kDisc>(w, a, p, in, t0 + kSBlock + lane, abort, spinLimit);
        if (!ok) break;
        p = fillLoadX<false, kDisc>(a, in, t0 + 2 * kSBlock + lane);
        __syncwarp();
        const int n = min(kSBlock, T - t0);
        int gA, gB;
        interiorRunS<8>(a, S, t0, n, gA, gB);
        int g = 0;
        RunX ip{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
        // the general steps before the interior ones (or all of them), then the interior, then the general ones after
#pragma unroll 1
        for (int part = 0; part < 2; ++part) {
            const bool inner = part == 0 && gB > gA;
            const int end = inner ? gA : n;
#pragma unroll 1
            for (; g < end; g += 8) {
                fwdStepX<MODE, 0, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 1, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 2, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 3, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 4, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 5, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 6, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 7, true, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
            }
            if (!inner) break;
            const int u0 = f.u;
            ip.col = w.s.col + (f.u & (kSWin - 1));
            ip.ring = w.s.ring + (f.u & (kSRingWin - 1));
            ip.cnt = w.cnt + (f.u & (kSRingWin - 1));
            ip.w1 = const_cast<float *>(f.w1src);
            ip.align = f.align;
            ip.out = out + 2 * (ptrdiff_t)(f.u - (R - 1));
#pragma unroll 1
            for (; g < gB; g += 8) {
                fwdStepX<MODE, 0, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 1, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 2, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 3, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 4, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 5, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 6, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                fwdStepX<MODE, 7, false, ANCH>(f, a, w, s, lane, row, M, out, x.anchorPart, ip);
                ip.col += 8;
                ip.ring += 8;
                ip.cnt += 8;
                ip.w1 -= 8 * SW;
                ip.align += 8 * SW;
                ip.out += 16;
            }
            f.u = u0 + (gB - gA);
            if (f.align != nullptr) f.align += (gB - gA) * SW;
            f.w1src -= (gB - gA) * SW;
            f.gAhead -= gB - gA;
        }
    }
    if (!kDisc) cpAsyncWait<0>();  // no copy outlives the sweep (the slots are reused)
    if (!ok) return false;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if (row + k > M) continue;
        if (kDisc) {
            x.rowMax[row + k] = f.rmax[k];
            x.rowCnt[row + k] = f.cnt;
        } else {
            foldBest(*exact, f.best[k].v, f.cSum[k]);
        }
    }
    return true;
}

__device__ __forceinline__ ExactBest warpBest(ExactBest b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        double m = __shfl_xor_sync(kFull, b.m, o);
        int e = __shfl_xor_sync(kFull, b.e, o);
        if (m != 0.0 && (b.m == 0.0 || e > b.e || (e == b.e && m > b.m))) {
            b.m = m;
            b.e = e;
        }
    }
    return b;
}

// Reference counts from the discovery maxima, scanned in the reference's row
// order (backward: M..0 from cnt[M+1] = 0; forward: 0..M, cnt[i+1] after row
// i).  One warp: 32 rows loaded at a time, the scan over shuffles.
template <bool BACKWARD>
__device__ __forceinline__ void exactScan(const float *rowMax, const int *rowCnt, int *cnt, int M, int lane) {
    if (lane == 0) cnt[BACKWARD ? M + 1 : 0] = 0;
    int c = 0;
    for (int r0 = 0; r0 <= M; r0 += kLanes) {
        const int q = r0 + lane, i = BACKWARD ? M - q : q;
        const bool on = q <= M;
        const float mx = on ? __ldcg(rowMax + i) : 0.0f;
        const int rc = on ? __ldcg(rowCnt + i) : 0;
        int mine = 0;
        for (int k = 0; k < kLanes; ++k) {
            int d = __shfl_sync(kFull, rc, k) - c;
            d = d > 15 ? 15 : (d < -15 ? -15 : d);
            // x 2^(64 d), exact: a power built from its exponent bits
            const double pre = (double)__shfl_sync(kFull, mx, k) *
                               __hiloint2double((1023 + kRescaleBits * d) << 20, 0);
            c += pre > (double)kRescaleThresh ? 1 : 0;
            if (lane == k) mine = c;
        }
        if (on) cnt[BACKWARD ? i : i + 1] = mine;
    }
}

// Pairs the fast kernel could not score exactly (a row maximum above
// RESCALE_THRESH in either sweep, a score beyond float range, or a mid
// product too small for a normal float), or every pair when force is set, go
// to the queue of the exact path.  queueCount[0] counts them.  With `only`,
// pairs whose entry is 0 are skipped.
__global__ void flagKernel(const PairOut *po, int n, int force, int *queue, int *queueCount, const uint8_t *only) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || (only && !only[k])) return;  // only: the pairs that have mid scores (search survivors)
    const PairOut o = po[k];
    const bool ok = !force && o.maxYb <= kRescaleThresh && o.maxFw <= kRescaleThresh && o.mid < INFINITY &&
                    o.filt < INFINITY && o.mid >= 0x1p-100f;
    if (!ok) queue[atomicAdd(queueCount, 1)] = k;
}

// Orders the exact-path queue costliest pair first ((M + 1) L cells, ties by
// pair position), so that the persistent CTAs that take pairs in queue order
// end on the cheapest ones, and the order no longer depends on the flag
// kernel's atomics.  One CTA of 1024 threads, a bitonic sort of up to
// kQueueSortMax entries in shared memory; a longer queue keeps its order.
constexpr int kQueueSortMax = 4096;
__global__ void __launch_bounds__(1024) queueSortKernel(int *queue, const int *queueCount, const DevPair *pairs) {
    __shared__ unsigned long long key[kQueueSortMax];
    const int cnt = *queueCount;
    if (cnt < 2 || cnt > kQueueSortMax) return;
    int n = 2;
    while (n < cnt) n *= 2;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        unsigned long long v = 0;  // padding sorts last
        if (i < cnt) {
            const int k = queue[i];
            const DevPair p = pairs[k];
            const long long cells = (long long)(p.M + 1) * p.L;
            const unsigned long long c = cells < 0xffffffffLL ? (unsigned long long)cells : 0xffffffffULL;
            // descending cost, then ascending position (complemented)
            v = (c << 32) | (unsigned long long)(0x7fffffffu - (unsigned)k);
        }
        key[i] = v;
    }
    __syncthreads();
    for (int size = 2; size <= n; size *= 2) {
        for (int stride = size / 2; stride > 0; stride /= 2) {
            for (int i = threadIdx.x; i < n / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const bool desc = (lo & size) == 0;  // the final merge (size == n) is descending
                const unsigned long long a = key[lo], b = key[hi];
                if (desc ? a < b : a > b) {
                    key[lo] = b;
                    key[hi] = a;
                }
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) queue[i] = (int)(0x7fffffffu - (unsigned)(key[i] & 0xffffffffULL));
}

// The traceback's row-major W0 and W1 (row i at i L) from the replay's steps: a
// tile of 128 steps of one stripe through shared memory, read and written in
// whole lines.  (The sweeps storing each cell in place made 64 four-byte
// stores a step, each in its own line: 4.6 ms for 55 hits of M = 400 x 2.2 kb.)
constexpr int kTileSteps = 128;
__global__ void __launch_bounds__(256) alignRowsKernel(const AlignJob *jobs, const float *steps, float *cells) {
    __shared__ float tile[kTileSteps][kExactStripe + 1];
    const AlignJob jb = jobs[blockIdx.z >> 1];
    const bool backward = (blockIdx.z & 1) != 0;
    const int s = blockIdx.y, nS = exactStripes(jb.M), t0 = blockIdx.x * kTileSteps, T = jb.L - 1 + kExactStripe;
    if (s >= nS || t0 >= T) return;
    const long long stripeFloats = pipeStripeFloats(jb.L, kExactRows);
    const float *src = steps + jb.stepOff + (backward ? nS + s : s) * stripeFloats + (size_t)t0 * kExactStripe;
    const int n = min(kTileSteps, T - t0);
    for (int q = threadIdx.x; q < n * kExactStripe; q += blockDim.x)
        tile[q / kExactStripe][q % kExactStripe] = __ldcs(src + q);
    __syncthreads();
    float *out = cells + 2 * jb.cellOff + (backward ? (size_t)(jb.M + 1) * jb.L : 0);
    for (int r = threadIdx.x >> 5; r < kExactStripe; r += blockDim.x >> 5) {
        const int i = s * kExactStripe + r, owner = r / kExactRows, k = r % kExactRows;
        if (i > jb.M) break;
        // the row's first column is at this step
        const int lag = backward ? (kLanes - 1 - owner) * kExactRows + (kExactRows - 1 - k) : r;
        for (int t = threadIdx.x & 31; t < n; t += kLanes) {
            const int u = t0 + t - lag;
            if (u >= 0 && u < jb.L) out[(size_t)i * jb.L + (backward ? jb.L - 1 - u : u)] = tile[t][r];
        }
    }
}

template <bool ANCH, bool ALIGN = false>
__global__ void __launch_bounds__(kExactMaxWarps * kLanes, 1) exactPipeKernel(ExactPipeArgs g) {
    extern __shared__ float4 smRaw[];
    __shared__ float smBg[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WindowX &wx = reinterpret_cast<WindowX *>(smRaw)[warp];
    const int C = clusterSize(), rank = clusterRank(), G = C * (blockDim.x >> 5);
    const int me = warp * C + rank;  // consecutive stripes on different CTAs
    const int cluster = blockIdx.x / C, nClusters = gridDim.x / C;
    float *base = g.pool + (size_t)cluster * g.poolSlot;
    unsigned long long *ring = g.ring + (size_t)cluster * g.ringSlot;
    int *abort = g.abort;
    const int n = *g.queueCount;
    for (int k = cluster; k < n; k += nClusters) {
        const int pi = g.queue[k];
        const DevPair p = g.pairs[pi];
        const DevProfile &pr = g.profiles[p.prof];
        const int nS = exactStripes(p.M);
        clusterSync(C);  // the previous pair's scratch, ring and background are done with
        if (warp == 0) smBg[lane] = lane < kNumCodes ? pr.bg[lane] : 0.0f;
        if (lane == 0) {
            PairCold &c = wx.s.cold;
            c.codes = g.codes + p.codeOff;
            c.pre = g.seeds + p.seedOff;
            c.suf = c.pre + p.L;
            c.coef = g.params + coefOffOf(pr.paramOff, pr.M);
            c.coefStride = pr.rowPad;
            c.smBg = smBg;
            c.sc = g.scales[pi];
            c.M = p.M;
        }
        __syncthreads();
        SweepArgs a;
        a.cold = &wx.s.cold;
        a.L = p.L;
        a.rowPad = kExactStripe;
        a.nS = 1;
        a.P = INT_MAX / 4;  // a stripe's sweep never reaches another stripe
        a.D = a.sFirst = 0;
        a.sStep = a.nMine = a.ringSlots = 1;
        a.ringStride = 0;
        a.ring = nullptr;
        a.alignOut = nullptr;
        ExactRows x;
        float *rows = base + exactW1Floats(p.M, p.L);
        float *maxB = rows, *maxF = rows + (p.M + 1);
        int *rcB = reinterpret_cast<int *>(maxF + (p.M + 1)), *rcF = rcB + (p.M + 1);
        x.cntB = rcF + (p.M + 1);
        x.cntF = x.cntB + (p.M + 2);
        double *bests = reinterpret_cast<double *>(
            base + (exactW1Floats(p.M, p.L) + 4LL * (p.M + 1) + 2LL * (p.M + 2) + 3) / 4 * 4);
        x.anchorPart = reinterpret_cast<float *>(bests + 4 * kPipeMaxCluster * kExactMaxWarps);
        const long long stripeFloats = pipeStripeFloats(p.L, kExactRows);
        // The stripe's emission rows in shared memory, and its W1.
        auto stripe = [&](int s) {
            __syncwarp();
            const float *src = g.emit + pr.emitOff + (size_t)s * kExactStripe + lane * kExactRows;
#pragma unroll
            for (int c = 0; c < kNumCodes; ++c)
                *reinterpret_cast<float2 *>(wx.emit + c * kExactStripe + lane * 2) =
                    __ldg(reinterpret_cast<const float2 *>(src + (size_t)c * pr.rowPad));
            __syncwarp();
            a.smE = wx.emit;
            a.w1 = base + s * stripeFloats;
        };
        unsigned long long *rb = ring, *rf = ring + 2LL * nS * p.L;  // boundary rows downward and upward
        const int sLast = nS - 1 >= me ? me + (nS - 1 - me) / G * G : -1;
        bool ok = abortPeek(abort) == 0;  // a wait ran out, in this kernel or before it: no pair is started
        ExactBest filt{0.0, 0}, mid{0.0, 0};
        // Stripe s hands its boundary row on through entry row s of a ring.
        auto backIn = [&](int s) { return s < nS - 1 ? rb + 2LL * (s + 1) * p.L : nullptr; };
        auto backOut = [&](int s) { return s > 0 ? rb + 2LL * s * p.L : nullptr; };
        auto foreIn = [&](int s) { return s > 0 ? rf + 2LL * (s - 1) * p.L : nullptr; };
        auto foreOut = [&](int s) { return s < nS - 1 ? rf + 2LL * s * p.L : nullptr; };
        // With twice as many warps as stripes the discovery sweeps run side by side.
        const bool twin = G >= 2 * nS;
        x.rowMax = maxB;
        x.rowCnt = rcB;
        for (int s = sLast; s >= 0 && ok; s -= G) {
            stripe(s);
            ok = exactBackward<kDiscover>(a, wx, s, lane, backIn(s), backOut(s), abort, g.spinLimit, x, nullptr);
        }
        x.rowMax = maxF;
        x.rowCnt = rcF;
        for (int s = twin ? me - nS : me; s < nS && ok; s += G) {
            if (s < 0) break;
            stripe(s);
            ok = exactForward<kDiscover, false>(a, wx, s, lane, foreIn(s), foreOut(s), abort, g.spinLimit, x, nullptr);
        }
        clusterSync(C);  // every row's maximum is written
        if (me == 0) exactScan<true>(maxB, rcB, x.cntB, p.M, lane);
        if (me == G - 1) exactScan<false>(maxF, rcF, x.cntF, p.M, lane);
        clusterSync(C);
        if (abortPeek(abort) != 0) ok = false;
        int *alignCnt = nullptr;
        float *alignW0 = nullptr;
        if (ALIGN && g.jobOf[pi] >= 0) {
            const AlignJob &jb = g.jobs[g.jobOf[pi]];
            alignW0 = g.alignSteps + jb.stepOff;
            alignCnt = g.alignRows + jb.rowOff;
        }
        for (int s = sLast; s >= 0 && ok; s -= G) {
            stripe(s);
            if (ALIGN && alignW0) a.alignOut = alignW0 + (nS + s) * stripeFloats;
            ok = exactBackward<kReplay>(a, wx, s, lane, backIn(s), backOut(s), abort, g.spinLimit, x, &filt);
        }
        for (int s = me; s < nS && ok; s += G) {
            stripe(s);
            if (ALIGN && alignW0) a.alignOut = alignW0 + s * stripeFloats;
            ok = exactForward<kReplay, ANCH>(a, wx, s, lane, foreIn(s), foreOut(s), abort, g.spinLimit, x, &mid);
        }
        filt = warpBest(filt);
        mid = warpBest(mid);
        if (lane == 0) {
            bests[4 * me] = filt.m;
            bests[4 * me + 1] = (double)filt.e;
            bests[4 * me + 2] = mid.m;
            bests[4 * me + 3] = (double)mid.e;
        }
        clusterSync(C);  // the bests, and with anchors the column partials, are written
        const int t = me * kLanes + lane, T = G * kLanes;
        const bool failed = abortPeek(abort) != 0;
        if (ALIGN && !failed && alignCnt != nullptr) {
            for (int i = t; i < p.M + 2; i += T) {
                alignCnt[i] = __ldcg(x.cntB + i);
                alignCnt[p.M + 2 + i] = __ldcg(x.cntF + i);
            }
        }
        if (ANCH && !failed && g.anchorOff[pi] >= 0) {
            // fold the stripes' partials of each column in row order
            const long long o = g.anchorOff[pi];
            for (int j = t; j < p.L; j += T) {
                float bm = 0.0f;
                int be = 0, br = 0;
                for (int s2 = 0; s2 < nS; ++s2) {
                    const float *pp = x.anchorPart + ((size_t)s2 * p.L + j) * 3;
                    const float cm = __ldcg(pp);
                    const int ce = __float_as_int(__ldcg(pp + 1));
                    if (xsLessMe(bm, be, cm, ce)) {
                        bm = cm;
                        be = ce;
                        br = __float_as_int(__ldcg(pp + 2));
                    }
                }
                g.anchorM[o + j] = bm;
                g.anchorE[o + j] = be;
                g.anchorRow[o + j] = br;
            }
        }
        if (me == 0) {
            ExactBest f{0.0, 0}, m{0.0, 0};
            auto fold = [](ExactBest &b, double vm, int ve) {
                if (vm != 0.0 && (b.m == 0.0 || ve > b.e || (ve == b.e && vm > b.m))) b = ExactBest{vm, ve};
            };
            for (int q = lane; q < G; q += kLanes) {
                fold(f, __ldcg(bests + 4 * q), (int)__ldcg(bests + 4 * q + 1));
                fold(m, __ldcg(bests + 4 * q + 2), (int)__ldcg(bests + 4 * q + 3));
            }
            f = warpBest(f);
            m = warpBest(m);
            if (lane == 0) {
                ExactOut o;
                o.mid = m.m == 0.0 ? xsZero() : XS{__double2float_rn(m.m), m.e};
                o.filt = f.m == 0.0 ? xsZero() : XS{__double2float_rn(f.m), f.e};
                o.failed = failed;
                g.out[pi] = o;
            }
        }
    }
    // no CTA of the cluster leaves while another may still read its part
    clusterSync(C);
}

}  // namespace dmst
