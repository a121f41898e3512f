// The plain schedule: one (read, profile) pair per kernel launch, the
// baseline the batched persistent kernel is measured against.  The launch is
// one CTA whose warps share the pair: its stripes (32 R profile rows each)
// are dealt to the warps round-robin and run as a stripe pipeline with
// the batched kernel's fast-path arithmetic.  A pair of
// nS stripes keeps min(nS, 8) warps busy, so its time is that of the one
// pair alone on the GPU, with none of the batching across pairs.  The
// results are those of the batched kernel bit for bit; a pair whose wait
// ran out is handed to the exact path (its mid is set to NaN, which the
// flag kernel routes there).
//
// Stripe pipeline.  Warp w runs stripes w, w + W, ... in processing order
// (top-down in the backward, bottom-up in the forward).  The rows crossing
// from stripe sp to sp+1 go through ring (sp mod 2W) in global memory.  Every
// warp publishes, in shared memory, how far its ring-writing lane has got
// (the position sp P' + column of the next column it computes), and before
// each refill of its staging window a warp waits until the stripe before
// each stripe it stages has written the ring columns the refill reads, and
// until the ring slot it is about to overwrite has been read.  Every wait is
// on a stripe earlier in processing order, and the stripe period P' = P + 128
// is long enough that a warp's window never reaches its next stripe before
// its current stripe's columns are all computed and published, so the waits
// cannot form a cycle.  Every wait is bounded: past the limit it sets the
// CTA's abort flag and all warps leave their sweeps at the next block.
#pragma once

#include "dp_exact_pipe.cuh"

namespace dmst {

constexpr int kPlainWarps = 8;       // warps of the CTA
constexpr int kPipeExtra = 128;      // stripe period P' = P + kPipeExtra
constexpr int kPipeSpinLimit = 1 << 24;  // default iterations of a wait (64 ns sleeps) before it gives up
static_assert(kPipeExtra >= kLanes - 1 + 2 * kBlock, "a window never reaches the next stripe early");

struct PipeSync {
    volatile int *progress;  // [kPlainWarps]: ring-writer position of each warp
    volatile int *abort;     // the CTA's abort flag
    int W;                   // warps running stripes
    int spinLimit;           // iterations of a wait before it gives up (sets the abort flag)
};

// Position of this warp's ring-writing lane (local time t0 - 31) at block
// boundary t0, and publication of it (after the lane's ring stores).
__device__ __forceinline__ int pipePos(const SweepArgs &a, int lt) {
    if (lt < 0) return a.sFirst * a.P;
    const int k = lt / a.P;
    if (k >= a.nMine) return INT_MAX;
    return (a.sFirst + k * a.sStep) * a.P + (lt - k * a.P);
}
__device__ __forceinline__ void pipePublish(const PipeSync &ps, int warp, int pos, int lane) {
    __threadfence_block();  // each lane's ring stores (lane 0 backward, lane 31 forward) ...
    __syncwarp();
    if (lane == 0) ps.progress[warp] = pos;  // ... before the position
}

// Lane 0 waits until warp w's position reaches target; false on abort.
__device__ __forceinline__ bool pipeWaitOne(const PipeSync &ps, int w, int target) {
    int it = 0;
    while (ps.progress[w] < target) {
        if (*ps.abort) return false;
        if (++it > ps.spinLimit) {
            *ps.abort = 1;
            return false;
        }
        __nanosleep(64);
    }
    return true;
}

// Before the block of local times [t0, t0 + kBlock) and the refill of the
// window entries [fill, fill + kBlock): the ring columns the refill reads are
// written, and the ring slots this block writes have been read.  Warp-uniform.
__device__ __forceinline__ bool pipeReady(const PipeSync &ps, const SweepArgs &a, int t0, int fill, int lane) {
    bool ok = true;
    if (lane == 0) {
        const int total = a.nMine * a.P;
        // readers: the last entry of each stripe the refill touches
        for (int u = fill; ok && u < fill + kBlock && u < total;) {
            const int k = u / a.P;
            const int kEnd = min(min(fill + kBlock, total), (k + 1) * a.P) - 1;  // last entry in stripe k
            const int sp = a.sFirst + k * a.sStep;
            const int jj = min(kEnd - k * a.P, a.L - 1);
            if (sp > 0 && u - k * a.P < a.L) ok = pipeWaitOne(ps, (sp - 1) % ps.W, (sp - 1) * a.P + jj + 1);
            u = (k + 1) * a.P;
        }
        // writers: before overwriting ring slot (sp mod 2W), stripe r = sp - 2W + 1 (which
        // reads the slot's previous contents) has staged all its columns: its writer lane
        // is past column L, and a warp's refills run at least 78 steps ahead of it
        for (int lt = max(t0 - (kLanes - 1), 0); ok && lt < t0 + kBlock - (kLanes - 1) && lt < total;) {
            const int k = lt / a.P;
            const int sp = a.sFirst + k * a.sStep;
            const int r = sp - a.ringSlots + 1;
            if (sp < a.nS - 1 && r >= 1) ok = pipeWaitOne(ps, r % ps.W, r * a.P + a.L);
            lt = (k + 1) * a.P;
        }
    }
    ok = __shfl_sync(kFull, ok, 0);
    __syncwarp();
    __threadfence_block();  // the positions seen before the refill's ring loads
    return ok;
}

// The sweeps of one warp in the stripe pipeline, with its share of the float
// maxima (filter best and largest Y in the backward, mid and largest W0 / Y0
// in the forward).
template <int R, bool MID>
__device__ bool backwardSweepPipe(const SweepArgs &a, Window &win, int warp, int lane, const PipeSync &ps,
                                  float &filtOut, float &maxYOut) {
    BwdState<R> b;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
        for (int k = 0; k < R; ++k) b.h[q][k] = b.z[q][k] = 0.0f;
        b.rb[q] = 0.0f;
    }
    b.sendW = b.sendY = b.filt = b.maxY = 0.0f;
    b.u = -(kLanes - 1 - lane);  // lane 31 leads
    b.sp = a.sFirst;
    b.jj = 0;
    b.wp = a.w1;
    const int total = a.nMine * a.P;
    const int T = (total + (kLanes - 1) + 2) / 3 * 3;
    if (!pipeReady(ps, a, -kBlock, 0, lane)) return false;
    fillBlock<true>(win, a, 0, lane);
    for (int t0 = 0; t0 < T; t0 += kBlock) {
        pipePublish(ps, warp, pipePos(a, t0 - (kLanes - 1)), lane);
        if (!pipeReady(ps, a, t0, t0 + kBlock, lane)) return false;
        fillBlock<true>(win, a, t0 + kBlock, lane);
        const int n = (t0 + kBlock < T ? kBlock : T - t0);
#pragma unroll 1
        for (int g = 0; g < n; g += 3) {
            backwardStep<R, MID, 0>(b, a, win, lane, total);
            backwardStep<R, MID, 1>(b, a, win, lane, total);
            backwardStep<R, MID, 2>(b, a, win, lane, total);
        }
    }
    pipePublish(ps, warp, INT_MAX, lane);
    filtOut = b.filt;
    maxYOut = b.maxY;
    return true;
}

template <int R>
__device__ bool forwardSweepPipe(const SweepArgs &a, Window &win, int warp, int lane, const PipeSync &ps,
                                 float &bestOut, float &maxOut) {
    FwdState<R> f;
#pragma unroll
    for (int h = 0; h < 3; ++h)
#pragma unroll
        for (int k = 0; k < R; ++k) f.w[h][k] = f.z[h][k] = 0.0f;
    f.sendIn = f.sendY = f.best = f.mx = 0.0f;
    f.u = -lane;  // lane 0 leads
    f.s = a.sFirst;
    f.j = 0;
    const int total = a.nMine * a.P;
    const int T = (total + (kLanes - 1) + 5) / 6 * 6;
    W1Stage<R> st{-lane, a.sFirst, 0};
#pragma unroll
    for (int k = 0; k < kW1Ahead; ++k) st.issue(a, win, k, lane, total);
    bool ok = pipeReady(ps, a, -kBlock, 0, lane);
    if (ok) fillBlock<false>(win, a, 0, lane);
    for (int t0 = 0; ok && t0 < T; t0 += kBlock) {
        pipePublish(ps, warp, pipePos(a, t0 - (kLanes - 1)), lane);
        ok = pipeReady(ps, a, t0, t0 + kBlock, lane);
        if (!ok) break;
        fillBlock<false>(win, a, t0 + kBlock, lane);
        const int n = (t0 + kBlock < T ? kBlock : T - t0);
#pragma unroll 1
        for (int g = 0; g < n; g += 6) {
            forwardStaged<R, 0>(f, a, win, lane, total, st);
            forwardStaged<R, 1>(f, a, win, lane, total, st);
            forwardStaged<R, 2>(f, a, win, lane, total, st);
            forwardStaged<R, 3>(f, a, win, lane, total, st);
            forwardStaged<R, 4>(f, a, win, lane, total, st);
            forwardStaged<R, 5>(f, a, win, lane, total, st);
        }
    }
    cpAsyncWait<0>();  // no copy outlives the sweep (the slots are reused)
    if (ok) pipePublish(ps, warp, INT_MAX, lane);
    bestOut = f.best;
    maxOut = f.mx;
    return ok;
}

// Scratch of one pair (floats): W1 of every stripe (nS x D x 32 R) and the
// 2W boundary rings of 4 P floats.
__host__ __device__ inline long long plainScratchFloats(int M, int L, int R) {
    const long long S = (long long)kLanes * R;
    const long long nS = (M + 1 + S - 1) / S;
    const long long Pw = wavePeriod(L);
    const long long D = Pw + kLanes - 1;
    const long long W = nS < kPlainWarps ? nS : kPlainWarps;
    return nS * D * S + 2LL * W * 4 * Pw;
}

template <int R, bool MID>
__global__ void __launch_bounds__(kPlainWarps * kLanes, 1)
    plainKernel(const DevPair *pairs, int pi, const DevProfile *profiles, const float *emit, const float *params,
                const uint8_t *codes, const float *seeds, const PairScales *scales, float *scratch, PairOut *out,
                int spinLimit) {
    extern __shared__ float4 smRaw[];
    Window *wins = reinterpret_cast<Window *>(smRaw);
    __shared__ float smBg[32];
    __shared__ int progress[kPlainWarps];
    __shared__ int abortFlag;
    __shared__ float part[4][kPlainWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const DevPair p = pairs[pi];
    const DevProfile &pr = profiles[p.prof];
    constexpr int S = kLanes * R;
    const int nS = (p.M + 1 + S - 1) / S;
    const int W = min(nS, kPlainWarps);
    Window &win = wins[warp];
    if (warp == 0) smBg[lane] = lane < kNumCodes ? pr.bg[lane] : 0.0f;
    if (threadIdx.x == 0) abortFlag = 0;
    if (lane == 0) {
        PairCold &c = win.cold;
        c.codes = codes + p.codeOff;
        c.pre = seeds + p.seedOff;
        c.suf = c.pre + p.L;
        c.coef = params + coefOffOf(pr.paramOff, pr.M);
        c.coefStride = pr.rowPad;
        c.smBg = smBg;
        c.sc = scales[pi];
        c.M = p.M;
    }
    PipeSync ps;
    ps.progress = progress;
    ps.abort = &abortFlag;
    ps.W = W;
    ps.spinLimit = spinLimit > 0 ? spinLimit : kPipeSpinLimit;
    SweepArgs a;
    a.cold = &win.cold;
    a.smE = emit + pr.emitOff;
    a.L = p.L;
    a.rowPad = pr.rowPad;
    a.nS = nS;
    const int Pw = wavePeriod(p.L);
    a.P = Pw + kPipeExtra;
    a.D = Pw + kLanes - 1;
    a.sFirst = warp;
    a.sStep = W;
    a.nMine = warp < W ? (nS - warp + W - 1) / W : 0;
    a.ringSlots = 2 * W;
    a.ringStride = 4LL * Pw;
    a.w1 = scratch;
    a.ring = scratch + (size_t)nS * a.D * S;
    a.alignOut = nullptr;
    float filt = 0.0f, maxY = 0.0f, mid = 0.0f, maxFw = 0.0f;
    bool ok = true;
    if (lane == 0) progress[warp] = warp < W ? pipePos(a, -1) : INT_MAX;
    __syncthreads();
    if (warp < W) ok = backwardSweepPipe<R, MID>(a, win, warp, lane, ps, filt, maxY);
    __syncthreads();  // every stripe's W1 is stored; the rings are free
    ok = ok && abortFlag == 0;
    if (MID) {
        if (lane == 0) progress[warp] = warp < W ? pipePos(a, -1) : INT_MAX;
        __syncthreads();
        if (warp < W && ok) ok = forwardSweepPipe<R>(a, win, warp, lane, ps, mid, maxFw);
        __syncthreads();
        ok = ok && abortFlag == 0;
    }
    filt = warpMax(filt);
    maxY = warpMax(maxY);
    mid = warpMax(mid);
    maxFw = warpMax(maxFw);
    if (lane == 0) {
        part[0][warp] = filt;
        part[1][warp] = maxY;
        part[2][warp] = mid;
        part[3][warp] = maxFw;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        PairOut o{0.0f, 0.0f, 0.0f, 0.0f};
        for (int w = 0; w < kPlainWarps; ++w) {
            o.filt = fmaxf(o.filt, part[0][w]);
            o.maxYb = fmaxf(o.maxYb, part[1][w]);
            o.mid = fmaxf(o.mid, part[2][w]);
            o.maxFw = fmaxf(o.maxFw, part[3][w]);
        }
        if (!ok) {  // a wait ran out: NaN results (the flag kernel queues a NaN mid for the exact path)
            o.mid = __int_as_float(0x7fc00000);
            o.filt = __int_as_float(0x7fc00000);
        }
        out[pi] = o;
    }
}

}  // namespace dmst
