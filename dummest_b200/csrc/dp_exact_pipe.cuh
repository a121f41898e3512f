// Exact row-rescaled DP for the pairs the fast kernels cannot score exactly (a
// row maximum above RESCALE_THRESH, or a product beyond float range): one pair
// on all warps of a CTA, or of a cluster of CTAs.
//
// The reference decides each row's rescale after the whole row is known
// (dummest-dp-backward.hh:560-573, dummest-dp-forward.hh:228-242), which a
// wavefront cannot wait for.  So each direction runs twice (the kDiscover
// and kReplay modes of the step functions in dp_wavefront.cuh):
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
// a barrier (neither reads the other's values), then the counts are scanned,
// then both replay sweeps.  Every wait is for an earlier stripe of the same
// cluster and bounded: a wait that runs out sets the cluster's abort flag,
// every warp leaves its sweep, and the pair and those after it on the cluster
// are marked failed.
//
// Bound: the latency of a step (the FP64 products and, in the replay, the
// rescale factors add to the fast path's chain), so two rows per lane on as
// many warps as there are stripes.  With four rows per lane on the 8 warps of
// one CTA, 128-row stripes two to a warp, three pairs of M = 2000 x 10 kb took
// 47 ms on three SMs.
#pragma once

#include "dp_exact.cuh"
#include "dp_pipe.cuh"
#include "dp_traceback_job.cuh"

namespace dmst {

constexpr int kExactRows = 2;  // rows per lane
constexpr int kExactStripe = kLanes * kExactRows;
constexpr int kExactMaxWarps = 16;
// Steps of a block: a window entry per lane at most, and whole groups of the
// step functions' three (six) phases.
constexpr int kXBlock = 30;
static_assert(kXBlock % 6 == 0 && kXBlock <= kLanes && 31 + 2 * kXBlock <= kWin, "window geometry");

struct WindowX {
    Window w;
    float emit[kNumCodes * kExactStripe];  // the stripe's emission rows, code-major
};

__host__ __device__ inline int exactStripes(int M) { return (M + kExactStripe) / kExactStripe; }
// Scratch of a cluster (floats): W1 by stripe and diagonal, row maxima and
// counts of both discovery sweeps, reference counts, the warps' bests, and
// with anchors the stripes' column partials.
__host__ __device__ inline long long exactW1Floats(int M, int L) {
    return (long long)exactStripes(M) * (L + kLanes - 1) * kExactStripe;
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
    int *abort;             // one flag per cluster, 0 between kernels
    ExactOut *out;
    // anchors: anchorOff[pair] >= 0 is the offset of its L columns
    const long long *anchorOff;
    float *anchorM;
    int *anchorE, *anchorRow;
    // traceback jobs (jobOf[pair] >= 0): the replay sweeps' row-major W0 and W1
    // before each row's rescale (at float offset 2 AlignJob::cellOff: W0 at
    // [0, (M+1) L), W1 after it) and the reference's rescale counts
    // (AlignJob::rowOff in alignRows: cntB at [0, M+2), cntF after it)
    const int *jobOf;
    const AlignJob *jobs;
    float *alignCells;
    int *alignRows;
    int spinLimit;          // polls of a wait before it gives up
};

// A lane's operands of one window entry, as loaded.
struct FillX {
    int code;
    float suf, pre;
    unsigned long long wy, cnt;
};

template <bool BACKWARD, bool DISCOVER>
__device__ __forceinline__ FillX fillLoadX(const SweepArgs &a, const unsigned long long *in, int first, int lane) {
    FillX f{kPad, 0.0f, 0.0f, 0ull, 0ull};
    const int u = first + lane;
    if (lane < kXBlock && u < a.L) {
        if (BACKWARD) {
            const int j = a.L - 1 - u;
            f.code = (j + 1 < a.L) ? (int)__ldg(a.codes() + j + 1) : kPad;
            f.suf = __ldg(a.suf() + j);
            f.pre = __ldg(a.pre() + j);
        } else {
            f.code = (u >= 2) ? (int)__ldg(a.codes() + u - 2) : kPad;
            f.pre = __ldg(a.pre() + u);
        }
        if (in) {
            f.wy = ringPeek(in + 2 * (size_t)u);
            if (DISCOVER) f.cnt = ringPeek(in + 2 * (size_t)u + 1);
        }
    }
    return f;
}

// The window entries of a block, once their ring values are there; false:
// given up.
template <bool BACKWARD, bool DISCOVER>
__device__ __forceinline__ bool fillStoreX(Window &w, const SweepArgs &a, FillX f, unsigned long long *in, int first,
                                           int lane, int *abort, int spinLimit) {
    const int u = first + lane;
    if (in) {
        int it = 0;
        auto empty = [&]() { return f.wy == kRingEmpty || (DISCOVER && f.cnt == kRingEmpty); };
        while (__any_sync(kFull, empty())) {
            if (empty()) {
                f.wy = ringPeek(in + 2 * (size_t)u);
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
        if (lane < kXBlock && u < a.L) {
            ringPut(in + 2 * (size_t)u, kRingEmpty);
            if (DISCOVER) ringPut(in + 2 * (size_t)u + 1, kRingEmpty);
        }
    }
    if (lane < kXBlock) {
        const int e = u & (kWin - 1);
        const float bg = a.smBg()[f.code], off = __int_as_float(f.code * a.rowPad);
        w.col[e] = BACKWARD ? make_float4(off, bg, f.suf, f.pre) : make_float4(off, bg * a.sc().sC, f.pre, 0.0f);
        w.ring[e] = make_float4(__uint_as_float((unsigned)f.wy), __uint_as_float((unsigned)(f.wy >> 32)),
                                __uint_as_float((unsigned)f.cnt), 0.0f);
    }
    return true;
}

// One stripe (b.sp = a.nS - 1 - s) of a backward sweep.
template <int MODE>
__device__ bool exactBackward(const SweepArgs &a, Window &win, int s, int lane, unsigned long long *in, int *abort,
                              int spinLimit, const ExactRows *x, ExactBest *exact) {
    constexpr int R = kExactRows;
    constexpr bool kDisc = MODE == kDiscover;
    BwdState<R, MODE> b;
    b.sendW = b.sendY = b.filt = b.maxY = 0.0f;
    b.sendC = b.cnt = 0;
    b.u = -(kLanes - 1 - lane);  // lane 31 leads
    b.sp = a.nS - 1 - s;
    b.jj = 0;
    backwardStart<R, MODE>(b, a, lane, s, x);
    const int total = a.L;
    const int T = (total + (kLanes - 1) + 2) / 3 * 3;
    __syncwarp();
    FillX f = fillLoadX<true, kDisc>(a, in, 0, lane);
    if (!fillStoreX<true, kDisc>(win, a, f, in, 0, lane, abort, spinLimit)) return false;
    f = fillLoadX<true, kDisc>(a, in, kXBlock, lane);
    for (int t0 = 0; t0 < T; t0 += kXBlock) {
        __syncwarp();
        if (!fillStoreX<true, kDisc>(win, a, f, in, t0 + kXBlock, lane, abort, spinLimit)) return false;
        f = fillLoadX<true, kDisc>(a, in, t0 + 2 * kXBlock, lane);
        __syncwarp();
        const int n = min(kXBlock, T - t0);
#pragma unroll 1
        for (int g = 0; g < n; g += 3) {
            backwardStep<R, MODE, 0, true, true, false>(b, a, win, lane, total, x, exact);
            backwardStep<R, MODE, 1, true, true, false>(b, a, win, lane, total, x, exact);
            backwardStep<R, MODE, 2, true, true, false>(b, a, win, lane, total, x, exact);
        }
    }
    return true;
}

// One stripe of a forward sweep.
template <int MODE, bool ANCH>
__device__ bool exactForward(const SweepArgs &a, Window &win, int s, int lane, unsigned long long *in, int *abort,
                             int spinLimit, const ExactRows *x, ExactBest *exact) {
    constexpr int R = kExactRows;
    constexpr bool kDisc = MODE == kDiscover;
    FwdState<R, MODE> f;
    f.sendIn = f.sendY = f.best = f.mx = 0.0f;
    f.sendC = f.cnt = 0;
    f.sendAM = 0.0f;
    f.sendAE = f.sendAR = 0;
    f.u = -lane;  // lane 0 leads
    f.s = s;
    f.j = 0;
    forwardStart<R, MODE>(f, a, lane, s, x);
    const int total = a.L;
    const int T = (total + (kLanes - 1) + 5) / 6 * 6;
    W1Stage<R, true> st{-lane, s, 0};
    if (MODE == kReplay) {
#pragma unroll
        for (int k = 0; k < kW1Ahead; ++k) st.issue(a, win, k, lane, total);
    }
    __syncwarp();
    FillX g = fillLoadX<false, kDisc>(a, in, 0, lane);
    bool ok = fillStoreX<false, kDisc>(win, a, g, in, 0, lane, abort, spinLimit);
    if (ok) g = fillLoadX<false, kDisc>(a, in, kXBlock, lane);
    for (int t0 = 0; ok && t0 < T; t0 += kXBlock) {
        __syncwarp();
        ok = fillStoreX<false, kDisc>(win, a, g, in, t0 + kXBlock, lane, abort, spinLimit);
        if (!ok) break;
        g = fillLoadX<false, kDisc>(a, in, t0 + 2 * kXBlock, lane);
        __syncwarp();
        const int n = min(kXBlock, T - t0);
#pragma unroll 1
        for (int q = 0; q < n; q += 6) {
            forwardStaged<R, MODE, 0, ANCH, true, true, false>(f, a, win, lane, total, st, x, exact);
            forwardStaged<R, MODE, 1, ANCH, true, true, false>(f, a, win, lane, total, st, x, exact);
            forwardStaged<R, MODE, 2, ANCH, true, true, false>(f, a, win, lane, total, st, x, exact);
            forwardStaged<R, MODE, 3, ANCH, true, true, false>(f, a, win, lane, total, st, x, exact);
            forwardStaged<R, MODE, 4, ANCH, true, true, false>(f, a, win, lane, total, st, x, exact);
            forwardStaged<R, MODE, 5, ANCH, true, true, false>(f, a, win, lane, total, st, x, exact);
        }
    }
    if (MODE == kReplay) cpAsyncWait<0>();  // no copy outlives the sweep (the slots are reused)
    return ok;
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

template <bool ANCH, bool ALIGN = false>
__global__ void __launch_bounds__(kExactMaxWarps * kLanes, 1) exactPipeKernel(ExactPipeArgs g) {
    extern __shared__ float4 smRaw[];
    __shared__ float smBg[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WindowX &wx = reinterpret_cast<WindowX *>(smRaw)[warp];
    Window &win = wx.w;
    const int C = clusterSize(), rank = clusterRank(), G = C * (blockDim.x >> 5);
    const int me = warp * C + rank;  // consecutive stripes on different CTAs
    const int cluster = blockIdx.x / C, nClusters = gridDim.x / C;
    float *base = g.pool + (size_t)cluster * g.poolSlot;
    unsigned long long *ring = g.ring + (size_t)cluster * g.ringSlot;
    int *abort = g.abort + cluster;
    const int n = *g.queueCount;
    for (int k = cluster; k < n; k += nClusters) {
        const int pi = g.queue[k];
        const DevPair p = g.pairs[pi];
        const DevProfile &pr = g.profiles[p.prof];
        const int nS = exactStripes(p.M);
        clusterSync(C);  // the previous pair's scratch, ring and background are done with
        if (warp == 0) smBg[lane] = lane < kNumCodes ? pr.bg[lane] : 0.0f;
        if (lane == 0) {
            PairCold &c = win.cold;
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
        a.cold = &win.cold;
        a.L = p.L;
        a.rowPad = kExactStripe;
        a.nS = nS;
        a.P = INT_MAX / 4;  // a stripe's sweep never reaches another stripe
        a.D = p.L + kLanes - 1;
        a.sFirst = 0;
        a.sStep = a.nMine = 1;
        a.ringSlots = nS;
        a.ringStride = 4LL * p.L;
        a.w1 = base;
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
        // The stripe's emission rows in shared memory, addressed by profile row.
        auto stripe = [&](int s) {
            __syncwarp();
            const float *src = g.emit + pr.emitOff + (size_t)s * kExactStripe + lane * kExactRows;
#pragma unroll
            for (int c = 0; c < kNumCodes; ++c)
                *reinterpret_cast<float2 *>(wx.emit + c * kExactStripe + lane * 2) =
                    __ldg(reinterpret_cast<const float2 *>(src + (size_t)c * pr.rowPad));
            __syncwarp();
            a.smE = wx.emit - s * kExactStripe;
        };
        unsigned long long *rb = ring, *rf = ring + 2LL * nS * p.L;  // boundary rows downward and upward
        const int sLast = nS - 1 >= me ? me + (nS - 1 - me) / G * G : -1;
        bool ok = abortPeek(abort) == 0;  // a wait of an earlier pair ran out: no later pair is started
        ExactBest filt{0.0, 0}, mid{0.0, 0};
        // Stripe s hands its row to the next through entry row sp of the
        // step functions' numbering (the processing order).
        auto backIn = [&](int s) { return s < nS - 1 ? rb + 2LL * (nS - 2 - s) * p.L : nullptr; };
        auto foreIn = [&](int s) { return s > 0 ? rf + 2LL * (s - 1) * p.L : nullptr; };
        a.ring = reinterpret_cast<float *>(rb);
        x.rowMax = maxB;
        x.rowCnt = rcB;
        for (int s = sLast; s >= 0 && ok; s -= G) {
            stripe(s);
            ok = exactBackward<kDiscover>(a, win, s, lane, backIn(s), abort, g.spinLimit, &x, nullptr);
        }
        a.ring = reinterpret_cast<float *>(rf);
        x.rowMax = maxF;
        x.rowCnt = rcF;
        for (int s = me; s < nS && ok; s += G) {
            stripe(s);
            ok = exactForward<kDiscover, false>(a, win, s, lane, foreIn(s), abort, g.spinLimit, &x, nullptr);
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
            alignW0 = g.alignCells + 2 * jb.cellOff;  // two floats per cell
            alignCnt = g.alignRows + jb.rowOff;
        }
        a.ring = reinterpret_cast<float *>(rb);
        if (alignW0) a.alignOut = alignW0 + (size_t)(p.M + 1) * p.L;
        for (int s = sLast; s >= 0 && ok; s -= G) {
            stripe(s);
            ok = exactBackward<kReplay>(a, win, s, lane, backIn(s), abort, g.spinLimit, &x, &filt);
        }
        a.ring = reinterpret_cast<float *>(rf);
        a.alignOut = alignW0;
        for (int s = me; s < nS && ok; s += G) {
            stripe(s);
            ok = exactForward<kReplay, ANCH>(a, win, s, lane, foreIn(s), abort, g.spinLimit, &x, &mid);
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
