// The stripe pipeline: one (read, profile) pair on all warps of a CTA, or of a
// cluster of CTAs, for calls with too few pairs to fill the GPU with one warp
// per pair (dp_stagger.cuh).
//
// A pair's stripes (32 R profile rows) are dealt round-robin to the G warps
// of the cluster: warp g runs profile stripes s with s mod G = g, downward in
// the backward sweep and upward in the forward, each as a sweep of L - 1 + 32 R
// staggered steps (the step functions of dp_stagger.cuh, so the same bits).
// W1 of a stripe is written and read by the same lanes.  A stripe's boundary
// row goes to the next stripe's warp through a ring in global memory, one
// 8-byte (W, Y) entry per column and boundary.
//
// The entries are their own flags: every entry holds kRingEmpty (a NaN that no
// arithmetic produces) until its writer stores the pair of values in one
// 64-bit store, and the reader, after it took the values, puts kRingEmpty
// back, so no fences and no progress counters are needed and the ring is
// empty again when the kernel ends.  The reader's lanes load a block's entries
// a block ahead and look at them when they are needed; only then do they wait.
// Every wait is for a stripe earlier in processing order, whose warp is in the
// same cluster and hence resident, so the waits cannot form a cycle; each is
// bounded (spinLimit polls), after which the warp raises the abort flag, every
// warp leaves its sweep at its next look at the ring, and the pair's scores are
// NaN (the flag kernel sends such a pair to the exact path).  The flag is the
// ring buffer's, not the cluster's: a warp that gives up leaves entries behind,
// and the next kernel, which may be queued already, cuts the buffer into other
// slots.  So no pair is started while the flag is up; the host empties the
// buffer and lowers it.
//
// Why: one warp takes nS (L + 3) steps per sweep at about 290 cycles (one busy
// warp per SM sub-partition), however empty the GPU is.  With G warps a sweep
// is about L + nS (32 R + 64) steps, and the four sub-partitions of every SM
// have work.  The figures behind the choice of schedule are at pipePlan
// (dmst_api.cu).
#pragma once

#include "dp_stagger.cuh"

namespace dmst {

constexpr unsigned long long kRingEmpty = ~0ull;
constexpr int kRingSpin = 1 << 24;   // default polls of one wait before it gives up (about 0.5 us each)
constexpr int kPipeMaxWarps = 16;
constexpr int kPipeMaxCluster = 8;   // CTAs of a cluster (portable size)

template <int R>
struct WindowP {
    WindowS<R> s;
    float emit[kNumCodes * kLanes * R];  // the stripe's emission rows, code-major
};

// One pair's buffers: W1 by stripe and step, then (W, Y) rings of the backward
// and the forward sweep, one per stripe boundary.
__host__ __device__ inline long long pipeStripes(int M, int R) { return (M + 1 + kLanes * R - 1) / (kLanes * R); }
__host__ __device__ inline long long pipeStripeFloats(int L, int R) {
    return ((long long)L - 1 + kLanes * R + kSW1Slots - 1) / kSW1Slots * kSW1Slots * (kLanes * stagLaneStride(R));
}
__host__ __device__ inline long long pipeW1Floats(int M, int L, int R) {
    return pipeStripes(M, R) * pipeStripeFloats(L, R);
}
__host__ __device__ inline long long pipeRingEntries(int M, int L, int R) { return 2 * pipeStripes(M, R) * L; }

struct PipeArgs {
    const int *list;      // pair positions, costliest first
    const int *nList;     // their number on the device (null: nPairs)
    int nPairs;
    const DevPair *pairs;
    const DevProfile *profiles;
    const float *emit, *params;
    const uint8_t *codes;
    const float *seeds;
    const PairScales *scales;
    float *w1;            // one slot per cluster
    long long w1Slot;     // floats
    unsigned long long *ring;
    long long ringSlot;   // entries
    int *abort;           // the ring buffer's flag, 0 while every entry is empty between kernels
    PairOut *out;         // zeroed
    int spinLimit;        // polls of a wait before it gives up
};

__device__ __forceinline__ unsigned long long ringPeek(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ringPut(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ int abortPeek(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

struct FillP {
    int code;
    float suf, pre;
    unsigned long long ring;
};

// Column operands of local time u (zero outside the read), and the ring entry
// of its column when the stripe has one before it.
template <bool BACKWARD>
__device__ __forceinline__ FillP fillLoadP(const SweepArgs &a, const unsigned long long *ringIn, int u) {
    FillP f{kPad, 0.0f, 0.0f, 0ull};
    if (u >= 0 && u < a.L) {
        if (BACKWARD) {
            const int j = a.L - 1 - u;
            f.code = (j + 1 < a.L) ? (int)__ldg(a.codes() + j + 1) : kPad;
            f.suf = __ldg(a.suf() + j);
            f.pre = __ldg(a.pre() + j);
        } else {
            f.code = (u >= 2) ? (int)__ldg(a.codes() + u - 2) : kPad;
            f.pre = __ldg(a.pre() + u);
        }
        if (ringIn) f.ring = ringPeek(ringIn + u);
    }
    return f;
}

// Waits until no lane's entry is empty, empties the entries, and stores the
// window entries.  False: given up.
template <bool BACKWARD, int R>
__device__ __forceinline__ bool fillStoreP(WindowS<R> &w, const SweepArgs &a, FillP f, unsigned long long *ringIn, int u,
                                           int *abort, int spinLimit) {
    if (ringIn) {
        int it = 0;
        while (__any_sync(kFull, f.ring == kRingEmpty)) {
            if (f.ring == kRingEmpty) f.ring = ringPeek(ringIn + u);
            if (++it > spinLimit || (it & 63) == 0) {
                const bool gone = it > spinLimit || abortPeek(abort) != 0;
                if (__any_sync(kFull, gone)) {
                    if (gone) *reinterpret_cast<volatile int *>(abort) = 1;
                    return false;
                }
            }
        }
        if (u >= 0 && u < a.L) ringPut(ringIn + u, kRingEmpty);
    }
    const FillRegs r{f.code, f.suf, f.pre, __uint_as_float((unsigned)f.ring), __uint_as_float((unsigned)(f.ring >> 32))};
    fillStoreS<BACKWARD, R>(w, a, r, u);
    return true;
}

template <bool BACKWARD, int R>
__device__ __forceinline__ bool fillPrologueP(WindowS<R> &w, const SweepArgs &a, unsigned long long *ringIn, int lane,
                                              int *abort, int spinLimit, FillP &next) {
    constexpr int S = kLanes * R;
    for (int v = -S + lane; v < 0; v += kLanes) fillStoreS<BACKWARD, R>(w, a, FillRegs{kPad, 0.0f, 0.0f, 0.0f, 0.0f}, v);
    if (!fillStoreP<BACKWARD, R>(w, a, fillLoadP<BACKWARD>(a, ringIn, lane), ringIn, lane, abort, spinLimit)) return false;
    next = fillLoadP<BACKWARD>(a, ringIn, kSBlock + lane);
    return true;
}

// One stripe of the backward sweep.  `a` holds the stripe as the only one (nS
// = 1), or as the first of two (nS = 2) when it hands its lowest row on.
template <int R, bool MID>
__device__ bool pipeBackward(const SweepArgs &a, WindowS<R> &win, int lane, unsigned long long *ringIn, int *abort,
                             int spinLimit, float &filt, float &maxY) {
    constexpr int S = kLanes * R;
    constexpr int SW = kLanes * stagLaneStride(R);
    BwdS<R> b;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < R; ++k) b.h[q][k] = b.z[q][k] = b.evH[q][k] = 0.0f;
        b.rb[q] = b.bgH[q] = b.sufH[q] = b.preH[q] = 0.0f;
    }
#pragma unroll
    for (int k = 0; k < R; ++k) b.yPrev[k] = 0.0f;
    b.sendW = b.sendY = 0.0f;
    b.filt = filt;
    b.maxY = maxY;
    b.u = -(kLanes - 1 - lane) * R;
    b.jj = b.u;
    b.sp = 0;
    b.wp = a.w1 + lane * stagLaneStride(R);
    const int rowBase = (a.nS - 1) * S + lane * R;
    loadBackwardCoef<R>(b.c, a, rowBase);
    b.eS = (unsigned)__cvta_generic_to_shared(a.smE + rowBase);
    b.eG = nullptr;
    const int T = (a.L - 1 + S + 3) / 4 * 4;
    __syncwarp();
    FillP pf;
    if (!fillPrologueP<true, R>(win, a, ringIn, lane, abort, spinLimit, pf)) return false;
    for (int t0 = 0; t0 < T; t0 += kSBlock) {
        __syncwarp();
        if (!fillStoreP<true, R>(win, a, pf, ringIn, t0 + kSBlock + lane, abort, spinLimit)) return false;
        pf = fillLoadP<true>(a, ringIn, t0 + 2 * kSBlock + lane);
        __syncwarp();
        const int n = min(kSBlock, T - t0);
        int gA, gB;
        interiorRunS<4>(a, S, t0, n, gA, gB);
        bwdBlockS<R, MID, true, true>(b, a, win, lane, n, gA, gB, lane == 0 && a.nS > 1);
    }
    filt = b.filt;
    maxY = b.maxY;
    return true;
}

// One stripe of the forward sweep; step t reads the backward's W1 group
// L - 2 + 32 R - t of the stripe.
template <int R>
__device__ bool pipeForward(const SweepArgs &a, WindowS<R> &win, int lane, unsigned long long *ringIn, int *abort,
                            int spinLimit, float &best, float &mx) {
    constexpr int S = kLanes * R;
    constexpr int SW = kLanes * stagLaneStride(R);
    FwdS<R> f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < R; ++k) f.w[q][k] = f.z[q][k] = f.evH[q][k] = 0.0f;
        f.bgH[q] = f.preH[q] = 0.0f;
    }
#pragma unroll
    for (int k = 0; k < R; ++k) f.ninPrev[k] = f.yPrev[k] = 0.0f;
    f.sendIn = f.sendY = 0.0f;
    f.best = best;
    f.mx = mx;
    f.u = -lane * R;
    f.jj = f.u;
    f.sp = 0;
    loadForwardCoef<R>(f.c, a, lane * R);
    f.eS = (unsigned)__cvta_generic_to_shared(a.smE + lane * R);
    f.eG = nullptr;
    const int steps = a.L - 1 + S;
    const int T = (steps + kSW1Slots - 1) / kSW1Slots * kSW1Slots;
    {
        const float *src = a.w1 + (size_t)(steps - 1) * SW + lane * stagLaneStride(R);
#pragma unroll
        for (int k = 0; k < kSW1Ahead; ++k) {
            cpAsyncStage<R>(&win.w1[k][lane * stagLaneStride(R)], src);
            cpAsyncCommit();
            src -= SW;
        }
        f.w1src = src;
        f.gAhead = steps - 1 - kSW1Ahead;
    }
    __syncwarp();
    FillP pf;
    bool ok = fillPrologueP<false, R>(win, a, ringIn, lane, abort, spinLimit, pf);
    for (int t0 = 0; ok && t0 < T; t0 += kSBlock) {
        __syncwarp();
        ok = fillStoreP<false, R>(win, a, pf, ringIn, t0 + kSBlock + lane, abort, spinLimit);
        if (!ok) break;
        pf = fillLoadP<false>(a, ringIn, t0 + 2 * kSBlock + lane);
        __syncwarp();
        const int n = min(kSBlock, T - t0);
        int gA, gB;
        interiorRunS<8>(a, S, t0, n, gA, gB);
        fwdBlockS<R, true, true>(f, a, win, lane, n, gA, gB, lane == kLanes - 1 && a.nS > 1);
    }
    cpAsyncWait<0>();  // no copy outlives the sweep (the staging slots are reused)
    best = f.best;
    mx = f.mx;
    return ok;
}

// The CTAs of the cluster (all of them run the same pairs) wait for each
// other; one CTA alone waits for its own warps.
__device__ __forceinline__ void clusterSync(int size) {
    if (size == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}
__device__ __forceinline__ int clusterRank() {
    int r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ int clusterSize() {
    int r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// max of non-negative floats (ordered like their bits)
__device__ __forceinline__ void atomicMaxPos(float *p, float v) {
    if (v > 0.0f) atomicMax(reinterpret_cast<int *>(p), __float_as_int(v));
}

template <int R, bool MID>
__global__ void __launch_bounds__(kPipeMaxWarps * kLanes, 1) pipeKernel(PipeArgs g) {
    extern __shared__ float4 smRaw[];
    WindowP<R> *wins = reinterpret_cast<WindowP<R> *>(smRaw);
    __shared__ float smBg[32];
    constexpr int S = kLanes * R;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = blockDim.x >> 5;
    const int C = clusterSize(), rank = clusterRank();
    const int cluster = blockIdx.x / C, nClusters = gridDim.x / C;
    const int G = C * W;
    // consecutive stripes on different CTAs, so that few stripes use every CTA
    const int me = warp * C + rank;
    WindowP<R> &wp = wins[warp];
    WindowS<R> &win = wp.s;
    float *w1 = g.w1 + (size_t)cluster * g.w1Slot;
    unsigned long long *ring = g.ring + (size_t)cluster * g.ringSlot;
    int *abort = g.abort;
    const int n = g.nList ? *g.nList : g.nPairs;
    for (int k = cluster; k < n; k += nClusters) {
        const int pi = g.list[k];
        const DevPair p = g.pairs[pi];
        const DevProfile &pr = g.profiles[p.prof];
        const int nS = (int)pipeStripes(p.M, R);
        clusterSync(C);  // the previous pair's ring and background are done with
        if (warp == 0) smBg[lane] = lane < kNumCodes ? pr.bg[lane] : 0.0f;
        if (lane == 0) {
            PairCold &c = win.cold;
            c.codes = g.codes + p.codeOff;
            c.pre = g.seeds + p.seedOff;
            c.suf = c.pre + p.L;
            c.coefStride = pr.rowPad;
            c.smBg = smBg;
            c.sc = g.scales[pi];
            c.M = p.M;
        }
        __syncthreads();
        const float *coef = g.params + coefOffOf(pr.paramOff, pr.M);
        const float *emit = g.emit + pr.emitOff;
        const long long stripeFloats = pipeStripeFloats(p.L, R);
        SweepArgs a;
        a.alignOut = nullptr;
        a.cold = &win.cold;
        a.L = p.L;
        a.rowPad = S;
        a.P = INT_MAX / 4;  // a stripe's sweep never reaches another stripe
        a.D = a.sFirst = 0;
        a.sStep = a.nMine = a.ringSlots = 1;
        a.ringStride = 0;
        // The stripe's emission rows and coefficient rows; `top`: rows before
        // them in the numbering of the step functions.
        auto stripe = [&](int s, int top) {
            __syncwarp();
            const float *src = emit + (size_t)s * S + lane * R;
#pragma unroll
            for (int c = 0; c < kNumCodes; ++c) {
                float v[R];
                loadRows<R>(v, src + (size_t)c * pr.rowPad);
#pragma unroll
                for (int q = 0; q < R; ++q) wp.emit[c * S + lane * R + q] = v[q];
            }
            if (lane == 0) win.cold.coef = coef + (long long)s * S - top;
            __syncwarp();
            a.smE = wp.emit - top;
            a.w1 = w1 + s * stripeFloats;
        };
        float filt = 0.0f, maxY = 0.0f, mid = 0.0f, maxFw = 0.0f;
        bool ok = abortPeek(abort) == 0;  // a wait ran out, in this kernel or before it: no pair is started
        const int sLast = nS - 1 >= me ? me + (nS - 1 - me) / G * G : -1;  // this warp's highest stripe
        for (int s = sLast; s >= 0 && ok; s -= G) {
            a.nS = s > 0 ? 2 : 1;
            stripe(s, (a.nS - 1) * S);
            a.ring = reinterpret_cast<float *>(ring + (long long)s * p.L);
            ok = pipeBackward<R, MID>(a, win, lane, s < nS - 1 ? ring + (long long)(s + 1) * p.L : nullptr, abort, g.spinLimit, filt,
                                      maxY);
        }
        if (MID) {
            unsigned long long *fr = ring + (long long)nS * p.L;
            for (int s = me; s < nS && ok; s += G) {
                a.nS = s < nS - 1 ? 2 : 1;
                stripe(s, 0);
                a.ring = reinterpret_cast<float *>(fr + (long long)s * p.L);
                ok = pipeForward<R>(a, win, lane, s > 0 ? fr + (long long)(s - 1) * p.L : nullptr, abort, g.spinLimit, mid,
                                    maxFw);
            }
        }
        filt = warpMax(filt);
        maxY = warpMax(maxY);
        mid = warpMax(mid);
        maxFw = warpMax(maxFw);
        if (lane == 0) {
            PairOut *o = g.out + pi;
            if (ok) {
                atomicMaxPos(&o->filt, filt);
                atomicMaxPos(&o->maxYb, maxY);
                atomicMaxPos(&o->mid, mid);
                atomicMaxPos(&o->maxFw, maxFw);
            } else {  // a NaN above every finite score
                atomicMax(reinterpret_cast<int *>(&o->mid), 0x7fc00000);
                atomicMax(reinterpret_cast<int *>(&o->filt), 0x7fc00000);
            }
        }
    }
    // no CTA of the cluster leaves while another may still read its part
    clusterSync(C);
}

}  // namespace dmst
