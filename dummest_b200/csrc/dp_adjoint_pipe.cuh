// The adjoint (dp_adjoint.cuh: log T, its gradient, posterior tables) with a
// pair's stripes on all warps of a CTA or a cluster of CTAs.
//
// The arithmetic of a cell is adjointKernel's, operation for operation, in
// FP64.  What differs:
//
//  - Scaling.  adjointKernel holds each 32-row stripe at a power-of-two offset
//    taken from the whole boundary row below it, so a stripe cannot start
//    before the one below it has ended.  Here every offset is 0: a pair whose
//    forward values stay below 2^kAdjTop needs none, and the values are then
//    the same bits (scaling by powers of two is exact).  A pair beyond is
//    marked after its forward sweep and left to adjointKernel; a backward
//    value beyond marks the call, which then runs on adjointKernel as a whole.
//  - Stripe pipeline.  Stripe s runs on warp s mod G of the cluster, in both
//    sweeps.  Boundary rows go through one (W, Y) entry per column and stripe
//    in global memory, filled with kAdjEmpty (a NaN that no arithmetic
//    produces) before the kernel, so that each value is its own flag; a
//    warp's reads run one 32-column block ahead, and its waits (bounded,
//    always for an earlier stripe of the same cluster) can form no cycle.
//  - Operands.  Codes, background and seeds of a block of columns are loaded
//    a block ahead and kept as doubles in a shared-memory window, the stripe's
//    33 emission rows in a shared table, where adjointKernel waits each step
//    for two dependent global loads and converts them.
//  - The forward store is [stripe][step][W0 | Y0 | Z0][lane], so that every
//    store is one 256-byte line (8-byte pieces 24 bytes apart before).
//
// Bound: the latency of a step's FP64 chain (seven dependent FMAs in the
// backward) when pairs are few, FP64 issue when they are many; the time per
// step is therefore bought with warps: up to 10 per SM (shared memory).
// Measured, adjointKernel against this one: 64 reads of 300-1200 nt, M = 200,
// 6.92 -> 0.70 ms; posteriors of 12 windows of 2-3 kb, M = 400, 44.0 -> 1.81 ms;
// 1,024 reads of 600-2400 nt, M = 400, checkpointed 41.8 -> 17.9 ms.
#pragma once

#include <climits>

#include "dp_adjoint.cuh"
#include "dp_pipe.cuh"

namespace dmst {

constexpr unsigned long long kAdjEmpty = ~0ull;
constexpr int kAdjTop = 800;                            // values from 2^kAdjTop on need the stripe offsets
constexpr int kAdjTopHi = (1023 + kAdjTop) << 20;       // ... as the high word of the double
constexpr int kAdjPipeWarps = 10;
enum AdjStatus { kAdjOk = 0, kAdjRange = 1, kAdjRedo = 2 };

// Doubles of a pair's forward store (full: every block; checkpointed: the
// lanes' states and two recompute buffers), each followed by the stripes'
// shares of T; and of its boundary rows, forward then backward.
__host__ __device__ __forceinline__ long long adjPipeFull(int M, int L) {
    return (long long)adjStripes(M) * (L + 31) * 96 + adjStripes(M);
}
// (Two recompute buffers per warp that can work on the pair at once.)
__host__ __device__ __forceinline__ long long adjPipeBufs(int M, int G) {
    return 2LL * kAdjCk * 96 * (adjStripes(M) < G ? adjStripes(M) : G);
}
__host__ __device__ __forceinline__ long long adjPipeStates(int M, int L) {
    return (long long)adjStripes(M) * adjChunks(L) * 32 * kAdjCkVals;
}
__host__ __device__ __forceinline__ long long adjPipeCkpt(int M, int L, int G) {
    return adjPipeStates(M, L) + adjPipeBufs(M, G) + adjStripes(M);
}
__host__ __device__ __forceinline__ long long adjPipeBound(int M, int L) { return 4LL * adjStripes(M) * L; }

// Shared memory of a warp.
struct alignas(16) AdjWin {
    double ring[kAdjRing][96];       // backward: forward blocks, copied kAdjAhead steps ahead
    double ge[kNumCodes][32];        // backward: emission sums of the stripe
    double fbg[128], fseed[128];     // forward: background x sC and prefix seed by column
    double fw[64], fy[64];           // forward: the row below the stripe
    double bbg[64], bseed[64];       // backward: background and suffix seed by column from the right (forward: the latter by column)
    double bw[32], by[32];           // backward: the row above the stripe
    double yb[64];                   // backward: Y0 of the row below
    float emit[kNumCodes][33];       // rows 32 s - 1 .. 32 s + 31
    int fcode[128], bcode[64];
};

struct AdjPipeArgs {
    const AdjointJob *jobs;
    int nJobs;
    const DevPair *pairs;
    const DevProfile *profiles;
    const float *emit, *params;
    const uint8_t *codes;
    const float *seeds;
    const PairScales *scales;
    double *fstore;
    unsigned long long *bstore;  // kAdjEmpty throughout
    double *grad;
    double *logT;
    double *post;
    int *status;                 // per job, AdjStatus, zeroed
    int *abort;                  // a wait of the launch ran out
    int spinLimit;               // polls of a wait before it gives up
};

// The pair as every stripe sees it.
struct AdjPair {
    int L, M, nS, rowPad;
    const uint8_t *cd;
    const float *pre, *suf, *E, *par, *bg;
    double sC, s1, s2;
    unsigned long long *fb, *bb;  // boundary entries: [stripe][column] x (W, Y)
    int *abort;
    int spinLimit;
};

__device__ __forceinline__ double asD(unsigned long long v) { return __longlong_as_double((long long)v); }

// A lane's boundary entry of one column (W, Y), as loaded.
struct AdjEntry {
    unsigned long long w, y;
};
__device__ __forceinline__ AdjEntry adjPeek(const unsigned long long *row, int col, bool on) {
    AdjEntry e{0ull, 0ull};
    if (on) {
        e.w = ringPeek(row + 2 * (size_t)col);
        e.y = ringPeek(row + 2 * (size_t)col + 1);
    }
    return e;
}
// Waits until no lane's entry is empty; false: given up.
__device__ __forceinline__ bool adjWaitEntry(AdjEntry &e, const unsigned long long *row, int col, const AdjPair &p) {
    int it = 0;
    while (__any_sync(kFull, e.w == kAdjEmpty || e.y == kAdjEmpty)) {
        if (e.w == kAdjEmpty || e.y == kAdjEmpty) e = adjPeek(row, col, true);
        if (++it > p.spinLimit || (it & 63) == 0) {
            const bool gone = it > p.spinLimit || abortPeek(p.abort) != 0;
            if (__any_sync(kFull, gone)) {
                *reinterpret_cast<volatile int *>(p.abort) = 1;
                return false;
            }
        }
    }
    return true;
}

// The stripe's emission rows (row index r of the table is row 32 s - 1 + r;
// rows before 0 and past the padding read as 0).
__device__ __forceinline__ void adjLoadEmit(AdjWin &w, const AdjPair &p, int s, int lane) {
    const int r0 = 32 * s - 1 + lane, r1 = 32 * s + 31;
#pragma unroll
    for (int c = 0; c < kNumCodes; ++c) {
        w.emit[c][lane] = r0 >= 0 && r0 < p.rowPad ? __ldg(p.E + (size_t)c * p.rowPad + r0) : 0.0f;
        if (lane == 0) w.emit[c][32] = r1 < p.rowPad ? __ldg(p.E + (size_t)c * p.rowPad + r1) : 0.0f;
    }
}

// Forward operands of column j.
struct AdjFCol {
    int code;
    float bg, pre;
};
__device__ __forceinline__ AdjFCol adjFCol(const AdjPair &p, int j) {
    AdjFCol c{kPad, 0.0f, 0.0f};
    if (j >= 0 && j < p.L) {
        c.code = j >= 2 ? (int)__ldg(p.cd + j - 2) : kPad;
        c.bg = __ldg(p.bg + c.code);
        c.pre = __ldg(p.pre + j);
    }
    return c;
}
__device__ __forceinline__ void adjPutFCol(AdjWin &w, const AdjPair &p, const AdjFCol &c, int j) {
    const int e = j & 127;
    w.fcode[e] = c.code;
    w.fbg[e] = (double)c.bg * p.sC;
    w.fseed[e] = (double)c.pre;
}

// A lane's row in the forward sweep (row 32 s + lane); rows past M have zero
// coefficients and no seed, and stay 0.
struct AdjFRow {
    double a0, a1, a2, b0, d0, eps, pEnter, pd1, pd2, rs;
};
__device__ __forceinline__ AdjFRow adjFRow(const AdjPair &p, int s, int lane) {
    AdjFRow r{0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int i = 32 * s + lane;
    if (i <= p.M) {
        const float *q = p.par + (size_t)i * kParamFloats;
        r.a0 = q[0];
        r.a1 = (double)q[1] * p.s1;
        r.a2 = (double)q[2] * p.s2;
        r.b0 = q[3];
        r.d0 = q[6];
        r.eps = q[9];
        r.rs = 1.0;
        if (i > 0) {
            const float *qp = q - kParamFloats;
            r.pEnter = (double)qp[10] * p.sC;
            r.pd1 = (double)qp[7] * p.s2;
            r.pd2 = (double)qp[8] * p.s1;
        }
    }
    return r;
}

// Forward step k of a stripe (lane l at column k - l), adjFwdStep's
// arithmetic.  Columns before the read give 0; columns past it give values
// that no column of the read depends on.
__device__ __forceinline__ void adjFStep(const AdjFRow &r, AdjHist &h, const AdjWin &w, int k, int lane, double &W0,
                                         double &Y0, double &Z0) {
    const int e = (k - lane) & 127;
    double uj = __shfl_up_sync(kFull, h.pubW, 1);
    double yPrev = __shfl_up_sync(kFull, h.pubY, 1);
    if (lane == 0) {
        uj = w.fw[k & 63];
        yPrev = w.fy[k & 63];
    }
    const double em = (double)w.emit[w.fcode[e]][lane];  // row i - 1
    const double win = fma(r.pEnter * em, h.u3, fma(r.pd1, h.u2, fma(r.pd2, h.u1, yPrev)));
    Z0 = w.fbg[e] * fma(r.a0, h.w3, r.b0 * h.z3);
    W0 = fma(r.a1, h.w1, fma(r.a2, h.w2, fma(w.fseed[e], r.rs, win + Z0)));
    Y0 = fma(r.d0, W0, r.eps * yPrev);
    h.w3 = h.w2; h.w2 = h.w1; h.w1 = W0;
    h.z3 = h.z2; h.z2 = h.z1; h.z1 = Z0;
    h.u3 = h.u2; h.u2 = h.u1; h.u1 = uj;
    h.pubW = W0;
    h.pubY = Y0;
}

// The forward sweep of stripe s: `store` takes the blocks (full) or the states
// (CKPT).  part: the stripe's share of T (this lane's columns); hi: the
// largest high word of a value.
template <bool CKPT>
__device__ bool adjForward(AdjWin &w, const AdjPair &p, int s, int lane, double *store, double &part, int &hi) {
    const int nSteps = p.L + 31;
    const AdjFRow r = adjFRow(p, s, lane);
    AdjHist h = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const unsigned long long *in = s > 0 ? p.fb + 2 * (size_t)(s - 1) * p.L : nullptr;
    unsigned long long *out = p.fb + 2 * (size_t)s * p.L;
    const bool writer = lane == 31 && s < p.nS - 1;
    __syncwarp();
    adjLoadEmit(w, p, s, lane);
    for (int q = 0; q < 3; ++q) adjPutFCol(w, p, AdjFCol{kPad, 0.0f, 0.0f}, lane + 32 * (q + 1));
    w.bseed[32 + lane] = 0.0;
    AdjFCol next = adjFCol(p, lane);
    AdjEntry ent = adjPeek(in, lane, in && lane < p.L);
    float suf = lane < p.L ? __ldg(p.suf + lane) : 0.0f;
    for (int k0 = 0; k0 < nSteps; k0 += 32) {
        if (in && !adjWaitEntry(ent, in, k0 + lane, p)) return false;
        __syncwarp();
        adjPutFCol(w, p, next, k0 + lane);
        w.fw[(k0 + lane) & 63] = asD(ent.w);
        w.fy[(k0 + lane) & 63] = asD(ent.y);
        w.bseed[(k0 + lane) & 63] = (double)suf;
        const int jn = k0 + 32 + lane;
        next = adjFCol(p, jn);
        ent = adjPeek(in, jn, in && jn < p.L);
        suf = jn < p.L ? __ldg(p.suf + jn) : 0.0f;
        __syncwarp();
        if (CKPT && k0 % kAdjCk == 0) {  // the state the recompute starts from
            double *ck = store + ((size_t)s * adjChunks(p.L) + k0 / kAdjCk) * 32 * kAdjCkVals + lane;
            const double v[kAdjCkVals] = {h.w1, h.w2, h.w3, h.z1, h.z2, h.z3, h.u1, h.u2, h.u3, h.pubW, h.pubY};
#pragma unroll
            for (int q = 0; q < kAdjCkVals; ++q) ck[32 * q] = v[q];
        }
        const int n = min(32, nSteps - k0);
        double *o = CKPT ? nullptr : store + ((size_t)s * nSteps + k0) * 96 + lane;
#pragma unroll 4
        for (int q = 0; q < n; ++q) {
            const int k = k0 + q, j = k - lane;
            double W0, Y0, Z0;
            adjFStep(r, h, w, k, lane, W0, Y0, Z0);
            hi = max(hi, max(__double2hiint(W0), __double2hiint(Y0)));
            part = fma(W0, w.bseed[j & 63], part);
            if (!CKPT) {
                o[0] = W0;
                o[32] = Y0;
                o[64] = Z0;
                o += 96;
            }
            if (writer && j >= 0 && j < p.L) {
                ringPut(out + 2 * (size_t)j, (unsigned long long)__double_as_longlong(W0));
                ringPut(out + 2 * (size_t)j + 1, (unsigned long long)__double_as_longlong(Y0));
            }
        }
    }
    return true;
}

// The backward sweep of stripe s with the gradient sums and posteriors.
// F: the forward blocks (full) or the states (CKPT, with this warp's two
// recompute buffers buf).  scale = 2^-te.
template <bool POST, bool CKPT>
__device__ bool adjBackward(AdjWin &w, const AdjPair &p, int s, int lane, const double *F, double *buf, double invT,
                            double scale, double *gP, double *gE, double *cellP, double *matchP, int &hi) {
    const int L = p.L, M = p.M, nSteps = L + 31, nCk = adjChunks(L);
    const int i = 32 * s + 31 - lane;
    const bool rowOK = i <= M;
    double enter = 0, d0 = 0, d1 = 0, d2 = 0, a0 = 0, a1 = 0, a2 = 0, b0 = 0, eps = 0, q10 = 0, rs = 0;
    if (rowOK) {
        const float *q = p.par + (size_t)i * kParamFloats;
        enter = (double)q[10] * p.sC;
        d0 = q[6];
        d1 = (double)q[7] * p.s2;
        d2 = (double)q[8] * p.s1;
        a0 = (double)q[0] * p.sC;
        a1 = (double)q[1] * p.s1;
        a2 = (double)q[2] * p.s2;
        b0 = (double)q[3] * p.sC;
        eps = q[9];
        q10 = q[10];
        rs = 1.0;
    }
    double gEnter = 0, gD0 = 0, gD1 = 0, gD2 = 0, gA0 = 0, gA1 = 0, gA2 = 0, gEps = 0, gB0 = 0;
    const bool below = s > 0;
    const unsigned long long *in = s < p.nS - 1 ? p.bb + 2 * (size_t)(s + 1) * L : nullptr;
    unsigned long long *out = p.bb + 2 * (size_t)s * L;
    const unsigned long long *fBelow = below ? p.fb + 2 * (size_t)(s - 1) * L : nullptr;
    __syncwarp();
    adjLoadEmit(w, p, s, lane);
#pragma unroll
    for (int c = 0; c < kNumCodes; ++c) w.ge[c][lane] = 0.0;
    w.bcode[32 + lane] = kPad;
    w.bbg[32 + lane] = w.bseed[32 + lane] = w.yb[32 + lane] = 0.0;
    w.bw[lane] = w.by[lane] = 0.0;

    // CKPT: forward steps [cc kAdjCk, ...) of this stripe from their state, into buffer cc & 1.
    auto recompute = [&](int cc) {
        const AdjFRow r = adjFRow(p, s, lane);
        const int k0 = cc * kAdjCk, k1 = min(k0 + kAdjCk, nSteps);
        const double *ck = F + ((size_t)s * nCk + cc) * 32 * kAdjCkVals + lane;
        AdjHist h = {ck[0],       ck[32],      ck[32 * 2], ck[32 * 3], ck[32 * 4], ck[32 * 5],
                     ck[32 * 6], ck[32 * 7], ck[32 * 8], ck[32 * 9], ck[32 * 10]};
        AdjFCol c[3];
        AdjEntry e[2];
#pragma unroll
        for (int q = 0; q < 3; ++q) c[q] = adjFCol(p, k0 - 32 + 32 * q + lane);
#pragma unroll
        for (int q = 0; q < 2; ++q) e[q] = adjPeek(fBelow, k0 + 32 * q + lane, below && k0 + 32 * q + lane < L);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 3; ++q) adjPutFCol(w, p, c[q], k0 - 32 + 32 * q + lane);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            w.fw[(k0 + 32 * q + lane) & 63] = asD(e[q].w);
            w.fy[(k0 + 32 * q + lane) & 63] = asD(e[q].y);
        }
        __syncwarp();
        double *o = buf + (size_t)(cc & 1) * kAdjCk * 96 + lane;
#pragma unroll 4
        for (int k = k0; k < k1; ++k) {
            double W0, Y0, Z0;
            adjFStep(r, h, w, k, lane, W0, Y0, Z0);
            o[0] = W0;
            o[32] = Y0;
            o[64] = Z0;
            o += 96;
        }
        __threadfence_block();
        __syncwarp();  // the buffer before the copies that read it
    };
    int curChunk = -1;
    auto issue = [&](int t) {  // the block of forward step t into the ring
        if (t >= 0) {
            if (CKPT && t / kAdjCk != curChunk) {  // t descends: each chunk once, in order
                curChunk = t / kAdjCk;
                recompute(curChunk);
            }
            double *dst = w.ring[t & (kAdjRing - 1)];
            const double *src = CKPT ? buf + ((size_t)((t / kAdjCk) & 1) * kAdjCk + t % kAdjCk) * 96
                                     : F + ((size_t)s * nSteps + t) * 96;
            adjCp16(dst + 2 * lane, src + 2 * lane);
            if (lane < 16) adjCp16(dst + 64 + 2 * lane, src + 64 + 2 * lane);
        }
        adjCommit();
    };
    const int t0 = L + 30;  // the forward step of backward step 0
#pragma unroll 1
    for (int d = 0; d < kAdjAhead; ++d) issue(t0 - d);
    // operands of column jj from the right: code, background and suffix seed,
    // the row above (W, Y), and Y0 of the row below
    struct Col {
        int code;
        float bg, suf;
        unsigned long long yb;
    };
    auto col = [&](int jj) {
        Col c{kPad, 0.0f, 0.0f, 0ull};
        if (jj < L) {
            const int j = L - 1 - jj;
            c.code = jj >= 1 ? (int)__ldg(p.cd + j + 1) : kPad;
            c.bg = __ldg(p.bg + c.code);
            c.suf = __ldg(p.suf + j);
            if (below) c.yb = ringPeek(fBelow + 2 * (size_t)j + 1);
        }
        return c;
    };
    Col next = col(lane);
    AdjEntry ent = adjPeek(in, lane, in && lane < L);
    double n1 = 0, n2 = 0, n3 = 0;     // row i+1 at j+1, j+2, j+3
    double c1 = 0, c2 = 0;             // own row at j+1, j+2
    double zz1 = 0, zz2 = 0, zz3 = 0;  // own Z at j+1, j+2, j+3
    double pubW = 0, pubY = 0;
    for (int k0 = 0; k0 < nSteps; k0 += 32) {
        if (in && !adjWaitEntry(ent, in, k0 + lane, p)) {
            adjWait<0>();
            return false;
        }
        __syncwarp();
        {
            const int e = (k0 + lane) & 63;
            w.bcode[e] = next.code;
            w.bbg[e] = (double)next.bg;
            w.bseed[e] = (double)next.suf;
            w.yb[e] = asD(next.yb);
            w.bw[lane] = asD(ent.w);
            w.by[lane] = asD(ent.y);
        }
        next = col(k0 + 32 + lane);
        ent = adjPeek(in, k0 + 32 + lane, in && k0 + 32 + lane < L);
        __syncwarp();
        const int n = min(32, nSteps - k0);
        const bool inside = k0 + 32 <= L;  // no lane is past the read's first column
#pragma unroll(CKPT ? 1 : 4)
        for (int q = 0; q < n; ++q) {
            const int k = k0 + q, jj = k - lane, t = t0 - k, e = jj & 63;
            issue(t - kAdjAhead);
            double nj = __shfl_up_sync(kFull, pubW, 1);
            double ynj = __shfl_up_sync(kFull, pubY, 1);
            if (lane == 0) {
                nj = w.bw[q];
                ynj = w.by[q];
            }
            adjWait<kAdjAhead - 1>();  // blocks t and t-1 are in
            __syncwarp();
            const int c = w.bcode[e];
            const double ec = (double)w.emit[c][32 - lane];
            const double zbg = zz3 * w.bbg[e];
            const double W = fma(n3 * ec, enter,
                                 fma(ynj, d0, fma(n2, d1, fma(n1, d2, fma(zbg, a0, fma(c2, a2, fma(c1, a1,
                                     w.bseed[e] * rs)))))));
            const double Y = fma(eps, ynj, W);
            const double Z = fma(b0, zbg, W);
            hi = max(hi, max(__double2hiint(W), __double2hiint(Y)));
            if (lane == 31 && jj >= 0 && jj < L) {  // row 32s: the boundary for the stripe below
                ringPut(out + 2 * (size_t)jj, (unsigned long long)__double_as_longlong(W));
                ringPut(out + 2 * (size_t)jj + 1, (unsigned long long)__double_as_longlong(Y));
            }
            // forward values of the cell: block t, lane 31-lane; Y0 of the row
            // below: block t-1, lane 30-lane (row 32s-1: its boundary row)
            const double *bt = w.ring[t & (kAdjRing - 1)];
            double wA = bt[31 - lane], zA = bt[64 + 31 - lane];
            double yA = lane < 31 ? w.ring[(t - 1) & (kAdjRing - 1)][32 + 30 - lane] : w.yb[e];
            if (!inside && jj >= L) wA = zA = yA = 0.0;
            const double me = wA * n3 * p.sC;  // d/d(enter * e) without the other factor
            if (!POST) {
                gEnter = fma(me, ec, gEnter);
                w.ge[c][lane] = fma(me, q10, w.ge[c][lane]);
                gD0 = fma(wA, ynj, gD0);
                gD1 = fma(wA, n2, gD1);
                gD2 = fma(wA, n1, gD2);
                gA0 = fma(wA, zbg, gA0);
                gA1 = fma(wA, c1, gA1);
                gA2 = fma(wA, c2, gA2);
                gEps = fma(yA, ynj, gEps);
                gB0 = fma(zA, zbg, gB0);
            }
            if (POST && rowOK && jj >= 0 && jj < L) {
                const int j = L - 1 - jj;
                cellP[(size_t)i * L + j] = (wA * W * invT) * scale;
                if (j + 3 < L) matchP[(size_t)i * L + j + 3] = (me * ec * q10 * invT) * scale;
                if (j < 3) matchP[(size_t)i * L + j] = 0.0;
            }
            n3 = n2; n2 = n1; n1 = nj;
            c2 = c1; c1 = W;
            zz3 = zz2; zz2 = zz1; zz1 = Z;
            pubW = W;
            pubY = Y;
        }
    }
    adjWait<0>();  // no copy outlives the stripe (the ring is reused)
    __syncwarp();
    // d log T = dT / T: each lane adds its row's sums (the per-base scale of
    // each coefficient applied here, once per row)
    if (!POST && rowOK) {
        double *g = gP + (size_t)i * kParamFloats;
        const double v[9] = {gA0 * p.sC, gA1 * p.s1, gA2 * p.s2, gB0 * p.sC, gD0, gD1 * p.s2, gD2 * p.s1, gEps, gEnter};
        const int slot[9] = {0, 1, 2, 3, 6, 7, 8, 9, 10};
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const double x = (v[k] * invT) * scale;
            if (x != 0.0) atomicAdd(g + slot[k], x);
        }
        double *gr = gE + (size_t)i * kNumCodes;
        for (int cc = 0; cc < kNumCodes; ++cc) {
            const double x = (w.ge[cc][lane] * invT) * scale;
            if (x != 0.0) atomicAdd(gr + cc, x);
        }
    }
    return true;
}

template <bool POST, bool CKPT>
__global__ void __launch_bounds__(kAdjPipeWarps * kLanes, 1) adjointPipeKernel(AdjPipeArgs g) {
    extern __shared__ float4 smRaw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    AdjWin &w = reinterpret_cast<AdjWin *>(smRaw)[warp];
    const int C = clusterSize(), G = C * (blockDim.x >> 5);
    const int me = warp * C + clusterRank();  // consecutive stripes on different CTAs
    const int nClusters = gridDim.x / C;
    bool ok = true;
    for (int ji = blockIdx.x / C; ji < g.nJobs; ji += nClusters) {
        const AdjointJob job = g.jobs[ji];
        const DevPair d = g.pairs[job.pair];
        const DevProfile &pr = g.profiles[d.prof];
        const PairScales sc = g.scales[job.pair];
        AdjPair p;
        p.L = d.L;
        p.M = d.M;
        p.nS = adjStripes(d.M);
        p.rowPad = pr.rowPad;
        p.cd = g.codes + d.codeOff;
        p.pre = g.seeds + d.seedOff;
        p.suf = p.pre + d.L;
        p.E = g.emit + pr.emitOff;
        p.par = g.params + pr.paramOff;
        p.bg = pr.bg;
        p.sC = sc.sC;
        p.s1 = sc.s1;
        p.s2 = sc.s2;
        p.fb = g.bstore + job.bOff;
        p.bb = p.fb + 2 * (size_t)p.nS * p.L;
        p.abort = g.abort;
        p.spinLimit = g.spinLimit;
        double *F = g.fstore + job.fOff;
        double *buf = F + adjPipeStates(d.M, d.L) + (size_t)me * 2 * kAdjCk * 96;
        double *parts = F + (CKPT ? adjPipeStates(d.M, d.L) + adjPipeBufs(d.M, G) : (long long)p.nS * (p.L + 31) * 96);
        // forward: the stripes' shares of T, or NaN for a stripe beyond the range
        for (int s = me; s < p.nS; s += G) {
            double part = 0.0;
            int hi = 0;
            if (ok) ok = adjForward<CKPT>(w, p, s, lane, F, part, hi);
            part = warpSumD(part);
            hi = __reduce_max_sync(kFull, hi);
            if (lane == 0) parts[s] = ok && hi < kAdjTopHi ? part : __longlong_as_double(0x7ff8000000000000ll);
        }
        clusterSync(C);  // every share and every boundary row is written
        double tm = 0.0;
        int te = 0;
        bool inRange = true;
        for (int s0 = 0; s0 < p.nS; s0 += 32) {
            const double v = s0 + lane < p.nS ? __ldcg(parts + s0 + lane) : 0.0;
            if (__any_sync(kFull, v != v)) inRange = false;
            for (int q = 0; q < min(32, p.nS - s0); ++q) dxAdd(tm, te, __shfl_sync(kFull, v, q), 0);
        }
        if (!(tm > 0.0) || te > kAdjTop || te < -kAdjTop) inRange = false;
        if (me == 0 && lane == 0) {
            g.logT[ji] = log(tm) + te * 0.6931471805599453;
            if (!inRange) g.status[ji] = kAdjRange;
        }
        if (!inRange) continue;  // the same on every warp of the cluster
        const double invT = 1.0 / tm, scale = ldexp(1.0, -te);
        double *gP = g.grad, *gE = g.grad + (size_t)(p.M + 2) * kParamFloats;
        double *cellP = POST ? g.post + job.pOff : nullptr;
        double *matchP = POST ? cellP + (size_t)(p.M + 1) * p.L : nullptr;
        int hi = 0;
        const int sLast = p.nS - 1 >= me ? me + (p.nS - 1 - me) / G * G : -1;
        for (int s = sLast; s >= 0 && ok; s -= G)
            ok = adjBackward<POST, CKPT>(w, p, s, lane, F, buf, invT, scale, gP, gE, cellP, matchP, hi);
        hi = __reduce_max_sync(kFull, hi);
        if (lane == 0 && hi >= ((1023 + 1000) << 20)) g.status[ji] = kAdjRedo;
    }
    clusterSync(C);
}

}  // namespace dmst
