// Per-pair null model on the device: the codon/frameshift background prefix
// and suffix probabilities, the whole-sequence null total, the per-base
// scales and the seed vectors that the DP consumes.
//
// Restates, for one sequence (single-lane semantics), the reference's
//   buildNullSuffix            dummest-dp-backward.hh:6-55
//   buildNullPrefixFirstCodon  dummest-dp-backward.hh:58-100
//   buildNullTotalAndScales    dummest-dp-backward.hh:103-129
//   buildNullSeedModels        dummest-dp-backward.hh:133-165
// with the exact score algebra of dummest-score.hh / dummest-batch.hh: each
// step rounds a double to a float mantissa exactly where the reference does,
// so the seeds are bit-identical to the reference's (up to the last-ulp
// behaviour of log2/exp2 in double, which feeds one float rounding).
// A sequence's per-lane result in the reference does not depend on the batch
// it was scored in (lanes past their length are forced to 0 or 1), so the
// single-sequence form is the reference's result for that lane.
#pragma once

#include "dp_common.cuh"

namespace dmst {

struct XS {  // ExpScore (dummest-score.hh:28-33)
    float m;
    int e;
};

__device__ __forceinline__ XS xsZero() { return XS{0.0f, 0}; }
__device__ __forceinline__ XS pow2Score(int e2) { return XS{0.5f, e2 + 1}; }  // dummest-score.hh:197-199

// splitNormalizedDouble (dummest-batch.hh:42-53); also normalizeScore's frexp
// for every non-subnormal double (products here never reach double
// subnormals).
__device__ __forceinline__ XS splitNorm(double x, int eAdd) {
    if (x == 0.0) return xsZero();
    unsigned long long u = (unsigned long long)__double_as_longlong(x);
    int ef = (int)((u >> 52) & 0x7FFULL);
    if (ef == 0x7FF) return XS{__double2float_rn(x), eAdd};
    if (ef == 0) return xsZero();
    double m = __longlong_as_double((long long)((u & 0xFFFFFFFFFFFFFULL) | (1022ULL << 52)));
    return XS{__double2float_rn(m), eAdd + ef - 1022};
}

// scaleScore / batchScaleScores (dummest-score.hh:155-160, dummest-batch.hh:114-130).
__device__ __forceinline__ XS scaleScore(XS a, double f) {
    if (a.m == 0.0f) return xsZero();
    if (!(f > 0.0) || !isfinite(f)) return xsZero();
    return splitNorm(__dmul_rn((double)a.m, f), a.e);
}

// addScores, the scalar form (dummest-score.hh:169-181).  ldexp(m, -d) for
// 0 <= d <= 60 is the product of m and the power 2^-d built from its exponent
// bits: both exact, so the same bits.
__device__ __forceinline__ XS scalarAdd(XS a, XS b) {
    if (a.m == 0.0f) return b;
    if (b.m == 0.0f) return a;
    const bool agebe = a.e >= b.e;
    const XS h = agebe ? a : b, l = agebe ? b : a;
    const int d = h.e - l.e;
    if (d > 60) return h;
    const double inv = __longlong_as_double((long long)(1023 - d) << 52);
    return splitNorm(__dadd_rn((double)h.m, __dmul_rn((double)l.m, inv)), h.e);
}

// batchMulScores with eFold = 0 (dummest-batch.hh:58-72).
__device__ __forceinline__ XS batchMul(XS a, XS b) {
    if (a.m == 0.0f || b.m == 0.0f) return xsZero();
    double p = __dmul_rn((double)a.m, (double)b.m);
    int e = a.e + b.e;
    if (p < 0.5) {
        p *= 2.0;
        e -= 1;
    }
    return XS{__double2float_rn(p), e};
}

// mulScores, the scalar form (dummest-score.hh:184-188).
__device__ __forceinline__ XS scalarMul(XS a, XS b) {
    if (a.m == 0.0f || b.m == 0.0f) return xsZero();
    return splitNorm(__dmul_rn((double)a.m, (double)b.m), a.e + b.e);
}

// scoreToFloatClamped (dummest-score.hh:224-230), FP32 engine: exponent capped
// at 120.  With the mantissa in [0.5, 1], m 2^e is a normal float for
// -125 <= e <= 120, where it is the exact product of m and the power of two
// built from its exponent bits; smaller exponents (subnormal or zero results)
// go through ldexpf.
__device__ __forceinline__ float packScore(XS a) {
    if (a.m == 0.0f) return 0.0f;
    const int e = a.e > 120 ? 120 : a.e;
    if (e >= -125) return __fmul_rn(a.m, __int_as_float((e + 127) << 23));
    return ldexpf(a.m, e);
}

// ---------------------------------------------------------------------------
// The recurrences' score algebra without double arithmetic, bit for bit the
// double forms of dummest-batch.hh: each of those rounds the exact result of
// one operation on two float mantissas to a float, so one correctly rounded
// float operation gives the same mantissa, and the same operation rounded
// toward zero tells on which side of a power of two the exact result lies
// (the reference tests the double before it rounds to float, so a mantissa
// that rounds up to a power of two keeps the smaller exponent).  A dependent
// step then costs about 12 cycles (multiply) or 25 (add), where the double
// forms with their conversions took several hundred for a column.
//
// A zero carries the exponent kZeroExp, so that it is never the larger
// operand of a sum.
// ---------------------------------------------------------------------------
constexpr int kZeroExp = -(1 << 28);

__device__ __forceinline__ void storeXS(XS *p, XS v) {  // 8-byte aligned
    *reinterpret_cast<float2 *>(p) = make_float2(v.m, __int_as_float(v.e));
}
__device__ __forceinline__ XS tagZero(XS a) { return XS{a.m, a.m == 0.0f ? kZeroExp : a.e}; }

// batchMulScores with eFold = 0 (dummest-batch.hh:58-72), and scaleScore by a
// float factor given as mantissa in [0.5, 1) and exponent
// (dummest-batch.hh:114-130): the product of two mantissas in [0.5, 1] is in
// [0.25, 1], doubled when the exact product is below 0.5.
__device__ __forceinline__ XS mulF(XS a, XS b) {
    const float p = __fmul_rn(a.m, b.m);
    const bool lt = __fmul_rz(a.m, b.m) < 0.5f;
    return XS{lt ? p + p : p, a.e + b.e - (lt ? 1 : 0)};
}

// batchAddScores (dummest-batch.hh:78-108).  The smaller mantissa times 2^-d
// (d <= 60) is an exact float; the double sum is exact for d <= 29, and for
// larger d the smaller term is below 2^-29, where both roundings return the
// larger mantissa.
__device__ __forceinline__ XS addF(XS a, XS b) {
    const bool ag = a.e >= b.e;
    const float mh = ag ? a.m : b.m, ml = ag ? b.m : a.m;
    const int eh = max(a.e, b.e), d = min(eh - min(a.e, b.e), 60);
    const float inv = __int_as_float((127 - d) << 23);
    const float s = __fmaf_rn(ml, inv, mh);
    const bool ge = __fmaf_rz(ml, inv, mh) >= 1.0f && ml != 0.0f;
    return XS{ge ? s * 0.5f : s, eh + (ge ? 1 : 0)};
}

// scaleScore (dummest-batch.hh:114-130) by a double factor f, 0 < f < 1 (0:
// the result is zero): the one product whose 53-bit rounding can differ from
// a direct rounding to float, so it stays in double.  The mantissa goes to
// double by moving its bits.
__device__ __forceinline__ XS scaleD(XS a, double f) {
    const unsigned b = __float_as_uint(a.m);
    const double am = __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
    const double x = __dmul_rn(am, f);
    const int hi = __double2hiint(x);
    const float m = __double2float_rn(__hiloint2double((hi & 0xFFFFF) | 0x3FE00000, __double2loint(x)));
    const bool nz = a.m != 0.0f && f != 0.0;
    return XS{nz ? m : 0.0f, nz ? a.e + (hi >> 20) - 1022 : kZeroExp};
}

// mulScores and addScores, the scalar forms (dummest-score.hh:169-188), which
// renormalise a product or sum of exactly 1 (the batch forms keep it) and
// return the larger operand unchanged past 60 binades.  Zeros carry kZeroExp.
__device__ __forceinline__ XS scalarMulF(XS a, XS b) {
    const float p = __fmul_rn(a.m, b.m), z = __fmul_rz(a.m, b.m);
    const bool lt = z < 0.5f, one = z >= 1.0f;
    return XS{lt ? p + p : (one ? 0.5f : p), a.e + b.e + (one ? 1 : 0) - (lt ? 1 : 0)};
}
__device__ __forceinline__ XS scalarAddF(XS a, XS b) {
    const bool ag = a.e >= b.e;
    const float mh = ag ? a.m : b.m, ml = ag ? b.m : a.m;
    const int eh = max(a.e, b.e), d = eh - min(a.e, b.e);
    const float inv = __int_as_float((127 - min(d, 60)) << 23);
    const float s = __fmaf_rn(ml, inv, mh);
    const bool far = d > 60, ge = !far && __fmaf_rz(ml, inv, mh) >= 1.0f;
    return XS{far ? mh : (ge ? s * 0.5f : s), eh + (ge ? 1 : 0)};
}

struct NullRates {
    double single;      // BACKGROUND_FRAMESHIFT_RATE (a float value)
    double dbl;         // BACKGROUND_FRAMESHIFT_RATE_2 (a float value)
};

// A frameshift emission rate as the recurrences use it.  The rates are float
// values, so the mantissa is exact.  A rate of 0 gives 2^-1023 of its operand
// (mantissa 0.5), as splitting a zero product's bits does.
struct RateF {
    XS f;
    bool zero;
};
__device__ __forceinline__ RateF rateF(double v) {
    RateF r;
    r.zero = v == 0.0;
    r.f = r.zero ? XS{0.5f, -1021} : splitNorm(v, 0);
    return r;
}
template <bool ZERO>
__device__ __forceinline__ XS scaleByRate(XS a, const RateF &r) {
    const XS v = mulF(a, r.f);
    if (ZERO && r.zero) return XS{a.m == 0.0f ? 0.0f : 0.5f, a.e - 1022};
    return v;
}

// Pairs of one job are scored by two warps, one lane per pair (the pairs of
// one read side by side, so that their codon loads are broadcasts): one warp
// runs the prefix recurrence and then the prefix seeds, the other the suffix
// recurrence and the suffix seeds.  The lanes run in lock step over the
// columns of the longest read, store the recurrences' values interleaved (one
// coalesced 256-byte store per column) and write their seeds through a
// shared-memory transpose, so that each store writes 32 consecutive seeds of
// one pair.
//
// Bound: the serial chain of a column (prefix or suffix: a rate product and
// two sums) in small calls, issue in large ones.  So a pass first runs in
// plain floats with one exponent per group of kNullGroup columns: every step
// of the algebra rounds to 24 bits wherever its operands lie, so within the
// float range the scaled values are the same bits, and a column's chain is a
// product and two sums of 4 cycles each instead of 80 with the exponents'
// own.  The range is checked (below); a pass that leaves it runs again in the
// algebra.
// Measured, with the chains and the seeds' power chains one after another on
// one warp in double; with two warps in the float algebra; and now: 200 reads
// of 3.1 kb 4.40, 0.78 and 0.26 ms; 16 of 10 kb 13.3, 2.35 and 0.94 ms; 128,000
// pairs of 150-3000 nt 5.3, 2.2 and 0.98 ms.
//
// Temporary ExpScores of one job: prefix and suffix values, [nullTmpRows][32]
// each, with room for the last group's columns past the longest read.
constexpr int kNullGroup = 16;
__host__ __device__ constexpr long long nullTmpRows(long long L) { return L + 1 + kNullGroup; }
__host__ __device__ constexpr long long nullTmpEntries(long long L) { return 2 * 32 * nullTmpRows(L); }

struct NullJob {
    int first;  // index of the job's first (longest) pair in the pair-index array
    int count;  // pairs in the job (<= 32)
};

constexpr int kNullWarps = 4;
constexpr int kNullJobs = kNullWarps / 2;  // jobs of a CTA at a time
constexpr int kNullAhead = 8;   // codes loaded ahead of the recurrences (kNullGroup in scaled floats)
constexpr int kNullChunk = 16;  // stored values loaded ahead of the seed chains

// Columns j0 .. j0+31 of the job's seeds: stage[c][p] holds column j0 + c of
// pair p; write pair p's columns with lanes over columns.  Eight pairs at a
// time, all loads before the stores (a pair past the count has length 0): 200
// reads of 3.1 kb take 0.26 ms so, 0.36 one by one.
__device__ __forceinline__ void flushSeeds(float (*stage)[33], float *const *dst, const int *len, int count, int j0,
                                           int lane) {
    __syncwarp();
    for (int p0 = 0; p0 < count; p0 += 8) {
        float *to[8], v[8];
        int n[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            to[q] = dst[p0 + q];
            n[q] = len[p0 + q];
            v[q] = stage[lane][p0 + q];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (j0 + lane < n[q]) to[q][j0 + lane] = v[q];
    }
    __syncwarp();
}

// The first three columns, which have no codon before them.
template <bool ZERO>
__device__ __forceinline__ void prefixHead(int Lmax, float bg0, XS *pfx, int lane, const RateF &sNE, const RateF &dNE,
                                           XS &p1, XS &p2, XS &p3) {
    const double frame = 1.0 / 3.0;
    p1 = p2 = p3 = XS{0.0f, kZeroExp};
    for (int i = 0; i < 3 && i < Lmax; ++i) {
        const XS codon = tagZero(i == 2 ? scaleScore(splitNorm((double)bg0, 0), frame)
                                        : scaleScore(pow2Score(i == 1 ? -4 : -2), frame));
        const XS zero{0.0f, kZeroExp};
        const XS q = addF(codon, addF(i > 0 ? scaleByRate<ZERO>(p1, sNE) : zero, i > 1 ? scaleByRate<ZERO>(p2, dNE) : zero));
        storeXS(pfx + i * 32 + lane, q);
        p3 = p2;
        p2 = p1;
        p1 = q;
    }
}

// Prefix recurrence (dummest-dp-backward.hh:58-100), i = 0 .. Lmax-1; a lane
// past its read's end computes values that nothing reads.
template <bool ZERO>
__device__ __forceinline__ void prefixPass(const uint8_t *cd, int L, int Lmax, const double *tab, float bg0, XS *pfx,
                                           int lane, const RateF &sNE, const RateF &dNE) {
    XS p1, p2, p3;
    prefixHead<ZERO>(Lmax, bg0, pfx, lane, sNE, dNE, p1, p2, p3);
    // the code of column i is that of position i - 2
    const int last = L - 1;
    int c[kNullAhead];
#pragma unroll
    for (int u = 0; u < kNullAhead; ++u) c[u] = cd[min(1 + u, last)];
    for (int i0 = 3; i0 < Lmax; i0 += kNullAhead) {
#pragma unroll
        for (int u = 0; u < kNullAhead; ++u) {
            const int i = i0 + u;
            if (i >= Lmax) break;
            const double f = tab[min(c[u], 25) * 32];
            c[u] = cd[min(i + kNullAhead - 2, last)];
            const XS codon = scaleD(p3, f);
            const XS q = addF(codon, addF(scaleByRate<ZERO>(p1, sNE), scaleByRate<ZERO>(p2, dNE)));
            storeXS(pfx + (size_t)i * 32 + lane, q);
            p3 = p2;
            p2 = p1;
            p1 = q;
        }
    }
}

// The last two columns, whose codon is the trailing amount.
template <bool ZERO>
__device__ __forceinline__ void suffixHead(int Lmax, double keep, XS *sfx, int lane, const RateF &sNE, const RateF &dNE,
                                           XS &s1, XS &s2, XS &s3) {
    const XS trailing = tagZero(splitNorm(0.5 * keep, 0));
    s1 = pow2Score(0);  // suffix[i+1], [i+2], [i+3]
    s2 = s3 = XS{0.0f, kZeroExp};
    for (int k = 0; k < 2 && k < Lmax; ++k) {
        const XS codon{trailing.m, trailing.e - 2 * (k + 1) + 1};
        const XS v = addF(codon, addF(scaleByRate<ZERO>(s1, sNE), scaleByRate<ZERO>(k > 0 ? s2 : pow2Score(2), dNE)));
        storeXS(sfx + k * 32 + lane, v);
        s3 = s2;
        s2 = s1;
        s1 = v;
    }
}

// Suffix recurrence (:6-55) from suffix[L] = 1 and suffix[L+1..L+3] = 0; step
// k is column i = L-1-k, stored at k.
template <bool ZERO>
__device__ __forceinline__ void suffixPass(const uint8_t *cd, int L, int Lmax, const double *tab, double keep, XS *sfx,
                                           int lane, const RateF &sNE, const RateF &dNE) {
    XS s1, s2, s3;
    suffixHead<ZERO>(Lmax, keep, sfx, lane, sNE, dNE, s1, s2, s3);
    const int last = L - 1;
    int c[kNullAhead];
#pragma unroll
    for (int u = 0; u < kNullAhead; ++u) c[u] = cd[max(last - 2 - u, 0)];
    for (int k0 = 2; k0 < Lmax; k0 += kNullAhead) {
#pragma unroll
        for (int u = 0; u < kNullAhead; ++u) {
            const int k = k0 + u;
            if (k >= Lmax) break;
            const double f = tab[min(c[u], 25) * 32];
            c[u] = cd[max(last - k - kNullAhead, 0)];
            const XS codon = scaleD(s3, f);
            const XS v = addF(codon, addF(scaleByRate<ZERO>(s1, sNE), scaleByRate<ZERO>(s2, dNE)));
            storeXS(sfx + (size_t)k * 32 + lane, v);
            s3 = s2;
            s2 = s1;
            s1 = v;
        }
    }
}

// The prefix or suffix pass in the score algebra (out of line: what follows a
// pass in scaled floats only rarely).
__device__ __noinline__ void algebraPass(const uint8_t *cd, int L, int Lmax, const double *tab, double keep, float bg0,
                                         XS *val, int lane, NullRates r, bool suffix) {
    const RateF sNE = rateF(r.single * 0.25), dNE = rateF(r.dbl * 0.0625);
    if (sNE.zero || dNE.zero) {
        if (suffix)
            suffixPass<true>(cd, L, Lmax, tab, keep, val, lane, sNE, dNE);
        else
            prefixPass<true>(cd, L, Lmax, tab, bg0, val, lane, sNE, dNE);
    } else if (suffix) {
        suffixPass<false>(cd, L, Lmax, tab, keep, val, lane, sNE, dNE);
    } else {
        prefixPass<false>(cd, L, Lmax, tab, bg0, val, lane, sNE, dNE);
    }
}

// ---------------------------------------------------------------------------
// The recurrences in floats scaled by 2^-E, E per lane and group of columns.
// Sums and products round alike at every scale, so a value is the algebra's
// as long as nothing that counts leaves the normal range.  At a group's start
// the largest of the three values carried is in [2^60, 2^61), and no column's
// value exceeds 1.4 times the largest before it (the rates are below 0.25 and
// 0.0625, the codon factor of a distribution below 1).  While every value is
// at least 2^-60 and at most 2^120,
// a term that falls below 2^-126 (and is flushed) is less than half a unit in
// the last place of the sum it goes into, or of the sum after that, and
// leaves it unchanged as the algebra's does.  A pass that meets another value
// (a zero, or an infinity from codon factors far above 1) reports it and is run
// again in the algebra.
// ---------------------------------------------------------------------------
constexpr float kScaledMin = 8.673617379884035e-19f;  // 2^-60
constexpr float kScaledMax = 1.329227995784916e36f;   // 2^120

struct Scaled3 {  // the values of the last three columns, times 2^-E
    float a, b, c;
    int E;
};
// 2^k for -126 <= k <= 127
__device__ __forceinline__ float pow2F(int k) { return __int_as_float((k + 127) << 23); }
__device__ __forceinline__ Scaled3 scaled3(XS a, XS b, XS c) {
    Scaled3 s;
    s.E = max(a.e, max(b.e, c.e)) - 61;
    s.a = a.m * pow2F(max(a.e - s.E, -126));
    s.b = b.m * pow2F(max(b.e - s.E, -126));
    s.c = c.m * pow2F(max(c.e - s.E, -126));
    return s;
}
__device__ __forceinline__ void rescale(Scaled3 &s) {
    const int k = 187 - (__float_as_int(fmaxf(s.a, fmaxf(s.b, s.c))) >> 23);
    const float f = pow2F(min(k, 127));
    s.a *= f;
    s.b *= f;
    s.c *= f;
    s.E -= k;
}
// (float)((double)v f) for a normal v: scaleScore's two roundings.
__device__ __forceinline__ float scaleF(float v, double f) {
    const unsigned b = __float_as_uint(v);
    return __double2float_rn(__dmul_rn(__hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29)), f));
}
// One column from the last three (a the newest): codon + (a sNE + b dNE).
__device__ __forceinline__ float scaledColumn(Scaled3 &s, double f, float sN, float dN, bool inside, float &least,
                                              float &most) {
    const float q = __fadd_rn(scaleF(s.c, f), __fadd_rn(__fmul_rn(s.a, sN), __fmul_rn(s.b, dN)));
    least = fminf(least, inside ? q : 1.0f);
    most = fmaxf(most, q);
    s.c = s.b;
    s.b = s.a;
    s.a = q;
    return q;
}

// The prefix (suffix) pass in scaled floats; false: to be run in the algebra.
__device__ __forceinline__ bool prefixScaled(const uint8_t *cd, int L, int Lmax, const double *tab, float bg0, XS *pfx,
                                             int lane, const RateF &sNE, const RateF &dNE) {
    XS p1, p2, p3;
    prefixHead<false>(Lmax, bg0, pfx, lane, sNE, dNE, p1, p2, p3);
    if (Lmax <= 3) return true;
    Scaled3 s = scaled3(p1, p2, p3);
    const float sN = sNE.f.m * pow2F(sNE.f.e), dN = dNE.f.m * pow2F(dNE.f.e);
    float least = L > 3 ? fminf(s.a, fminf(s.b, s.c)) : 1.0f, most = 0.0f;
    const int last = L - 1;
    int c[kNullGroup];
#pragma unroll
    for (int u = 0; u < kNullGroup; ++u) c[u] = cd[min(1 + u, last)];
    XS *out = pfx + 3 * 32 + lane;
#pragma unroll 1
    for (int i0 = 3; i0 < Lmax; i0 += kNullGroup, out += kNullGroup * 32) {
        rescale(s);
#pragma unroll
        for (int u = 0; u < kNullGroup; ++u) {
            const double f = tab[min(c[u], 25) * 32];
            c[u] = cd[min(i0 + u + kNullGroup - 2, last)];
            const float q = scaledColumn(s, f, sN, dN, i0 + u < L, least, most);
            storeXS(out + u * 32, XS{q, s.E});
        }
    }
    return !__any_sync(kFull, !(least >= kScaledMin && most <= kScaledMax));
}

__device__ __forceinline__ bool suffixScaled(const uint8_t *cd, int L, int Lmax, const double *tab, double keep, XS *sfx,
                                             int lane, const RateF &sNE, const RateF &dNE) {
    XS s1, s2, s3;
    suffixHead<false>(Lmax, keep, sfx, lane, sNE, dNE, s1, s2, s3);
    if (Lmax <= 2) return true;
    Scaled3 s = scaled3(s1, s2, s3);
    const float sN = sNE.f.m * pow2F(sNE.f.e), dN = dNE.f.m * pow2F(dNE.f.e);
    float least = L > 2 ? fminf(s.a, fminf(s.b, s.c)) : 1.0f, most = 0.0f;
    const int last = L - 1;
    int c[kNullGroup];
#pragma unroll
    for (int u = 0; u < kNullGroup; ++u) c[u] = cd[max(last - 2 - u, 0)];
    XS *out = sfx + 2 * 32 + lane;
#pragma unroll 1
    for (int k0 = 2; k0 < Lmax; k0 += kNullGroup, out += kNullGroup * 32) {
        rescale(s);
#pragma unroll
        for (int u = 0; u < kNullGroup; ++u) {
            const double f = tab[min(c[u], 25) * 32];
            c[u] = cd[max(last - k0 - u - kNullGroup, 0)];
            const float q = scaledColumn(s, f, sN, dN, k0 + u < L, least, most);
            storeXS(out + u * 32, XS{q, s.E});
        }
    }
    return !__any_sync(kFull, !(least >= kScaledMin && most <= kScaledMax));
}

// A mantissa back to [0.5, 1) and its exponent to e.
__device__ __forceinline__ void renormF(float &m, int &e) {
    const int b = __float_as_int(m);
    e += (b >> 23) - 126;
    m = __int_as_float((b & 0x7FFFFF) | 0x3F000000);
}

// The seeds' power at the last column, base^(L-1) by rounded products.
__device__ __forceinline__ XS powerScaled(XS base, int L, int Lmax) {
    const int Lmin = __reduce_min_sync(kFull, L);
    float m = 0.5f;
    int e = 1 + (L - 1) * base.e;
    for (int k0 = 1; k0 < Lmax; k0 += kNullGroup) {
        if (k0 + kNullGroup <= Lmin) {
#pragma unroll
            for (int u = 0; u < kNullGroup; ++u) m = __fmul_rn(m, base.m);
        } else {
#pragma unroll
            for (int u = 0; u < kNullGroup; ++u)
                if (k0 + u < L) m = __fmul_rn(m, base.m);
        }
        renormF(m, e);
    }
    return XS{m, e};
}

// The seeds of columns 0 .. Lmax-1 (dummest-dp-backward.hh:137-164): stored
// value times a running power, the values of kNullChunk columns loaded while
// the ones before are used.  SUFFIX: column j's value is suffix[j+1], stored
// at L-2-j (1 at the last column).
template <bool SUFFIX>
__device__ __forceinline__ void seedPass(const XS *val, int L, int Lmax, XS run, XS step, float (*stage)[33],
                                         float *const *dst, const int *len, int count, int lane) {
    auto load = [&](int j) -> XS {
        const int q = SUFFIX ? L - 2 - j : j;
        if (SUFFIX ? j >= L - 1 : j >= L) return pow2Score(0);
        const float2 t = *reinterpret_cast<const float2 *>(val + (size_t)q * 32 + lane);
        return XS{t.x, __float_as_int(t.y)};
    };
    XS next[kNullChunk];
#pragma unroll
    for (int u = 0; u < kNullChunk; ++u) next[u] = load(u);
    for (int j0 = 0; j0 < Lmax; j0 += kNullChunk) {
        XS v[kNullChunk];
#pragma unroll
        for (int u = 0; u < kNullChunk; ++u) {
            v[u] = next[u];
            next[u] = load(j0 + kNullChunk + u);
        }
#pragma unroll
        for (int u = 0; u < kNullChunk; ++u) {
            stage[(j0 & 16) + u][lane] = packScore(mulF(v[u], run));
            run = mulF(run, step);
        }
        if ((j0 & 16) || j0 + kNullChunk >= Lmax) flushSeeds(stage, dst, len, count, j0 & ~31, lane);
    }
}

// The same from scaled values, the power's mantissa a chain of float products
// and its exponent counted beside it.  A seed in [2^-126, 2^119) converts by a
// shift of its exponent; a chunk with others is converted once more by
// packScore, whose cap takes the mantissa as the algebra holds it: 1 where a
// product below a power of two rounds up to it.  False: a product that is a
// power of two beyond the cap, whose mantissa depends on its factors' forms.
template <bool SUFFIX>
__device__ __forceinline__ bool seedScaled(const XS *val, int L, int Lmax, XS run, XS step, float (*stage)[33],
                                           float *const *dst, const int *len, int count, int lane) {
    auto load = [&](int j) -> XS {
        const int q = SUFFIX ? L - 2 - j : j;
        if (SUFFIX ? j >= L - 1 : j >= L) return XS{SUFFIX && j == L - 1 ? 0.5f : 0.0f, 1};
        const float2 t = *reinterpret_cast<const float2 *>(val + (size_t)q * 32 + lane);
        return XS{t.x, __float_as_int(t.y)};
    };
    bool bad = false;
    XS next[kNullChunk];
#pragma unroll
    for (int u = 0; u < kNullChunk; ++u) next[u] = load(u);
#pragma unroll 1
    for (int j0 = 0; j0 < Lmax; j0 += kNullChunk) {
        XS v[kNullChunk];
#pragma unroll
        for (int u = 0; u < kNullChunk; ++u) {
            v[u] = next[u];
            next[u] = load(j0 + kNullChunk + u);
        }
        XS r = run;
        int lo = 1, hi = 1;  // biased exponents of the seeds
#pragma unroll
        for (int u = 0; u < kNullChunk; ++u) {
            const float t = __fmul_rn(v[u].m, run.m);
            const int b = __float_as_int(t), ex = v[u].e + run.e;
            const int be = b == 0 ? 1 : (b >> 23) + ex;
            lo = min(lo, be);
            hi = max(hi, be);
            stage[(j0 & 16) + u][lane] = __int_as_float(b + (ex << 23));
            run.m = __fmul_rn(run.m, step.m);
            run.e += step.e;
        }
        renormF(run.m, run.e);
        if (lo < 1 || hi > 245) {
#pragma unroll
            for (int u = 0; u < kNullChunk; ++u) {
                XS t{__fmul_rn(v[u].m, r.m), v[u].e + r.e};
                if (t.m != 0.0f) {
                    const bool up = __fmul_rz(v[u].m, r.m) < t.m;
                    renormF(t.m, t.e);
                    if (t.e > 119 && t.m == 0.5f) {
                        bad = bad || !up;
                        t = XS{1.0f, t.e - 1};
                    }
                    stage[(j0 & 16) + u][lane] = packScore(t);
                }
                r.m = __fmul_rn(r.m, step.m);
                r.e += step.e;
            }
        }
        if ((j0 & 16) || j0 + kNullChunk >= Lmax) flushSeeds(stage, dst, len, count, j0 & ~31, lane);
    }
    return !__any_sync(kFull, bad);
}

__global__ void __launch_bounds__(kNullWarps * 32) nullModelKernel(const NullJob *jobs, int nJobs, const int *jobPairs,
                                                                   const DevPair *pairs, const DevProfile *profiles,
                                                                   const uint8_t *codes, float *seeds, XS *tmp,
                                                                   const long long *tmpOff, PairScales *scales,
                                                                   NullRates r) {
    __shared__ float stageAll[kNullWarps][32][33];
    __shared__ double tabAll[kNullJobs][26][32];  // a lane's codon factor by code: background x keep, 0 past code 24
    __shared__ float *dstAll[kNullWarps][32];
    __shared__ int lenAll[kNullWarps][32];
    __shared__ XS baseAll[kNullJobs][2][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int jw = warp >> 1;                    // the job of this warp pair
    const bool suffixWarp = (warp & 1) != 0;
    auto pairSync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + jw) : "memory"); };
    float (*stage)[33] = stageAll[warp];
    const double keep = 1.0 - r.single - r.dbl;      // codonKeepProbability
    const RateF sNE = rateF(r.single * 0.25);        // singleNucleotideEmission
    const RateF dNE = rateF(r.dbl * 0.0625);         // doubleNucleotideEmission
    const bool anyZero = sNE.zero || dNE.zero;
    const bool inRange = !anyZero && min(sNE.f.e, dNE.f.e) >= -60 && max(sNE.f.e, dNE.f.e) <= -1;
    for (int ji = blockIdx.x * kNullJobs + jw; ji < nJobs; ji += gridDim.x * kNullJobs) {
        const NullJob job = jobs[ji];
        const bool on = lane < job.count;
        const int pi = jobPairs[job.first + (on ? lane : 0)];
        const DevPair p = pairs[pi];
        const int L = p.L;
        const int Lmax = __shfl_sync(kFull, L, 0);
        const uint8_t *cd = codes + p.codeOff;
        const float *bg = profiles[p.prof].bg;
        float *pre = seeds + p.seedOff;
        dstAll[warp][lane] = suffixWarp ? pre + L : pre;
        lenAll[warp][lane] = on ? L : 0;
        XS *val = tmp + tmpOff[ji] + (suffixWarp ? 32 * (size_t)nullTmpRows(Lmax) : 0);
        pairSync();  // the previous job's table and bases are no longer read
        // each warp of the pair fills half of the table (scaleScore gives zero
        // for a factor that is not positive and finite)
#pragma unroll
        for (int c = 0; c < 13; ++c) {
            const int code = 2 * c + (suffixWarp ? 1 : 0);
            const double f = __dmul_rn(code < kNumCodes ? (double)bg[code] : 0.0, keep);
            tabAll[jw][code][lane] = f > 0.0 && isfinite(f) ? f : 0.0;
        }
        pairSync();
        const double *tab = &tabAll[jw][0][lane];
        const float bg0 = bg[cd[0]];
        const bool scaled = inRange && (suffixWarp ? suffixScaled(cd, L, Lmax, tab, keep, val, lane, sNE, dNE)
                                                   : prefixScaled(cd, L, Lmax, tab, bg0, val, lane, sNE, dNE));
        if (!scaled) algebraPass(cd, L, Lmax, tab, keep, bg0, val, lane, r, suffixWarp);
        if (!suffixWarp) {
            // Total and scales (dummest-dp-backward.hh:103-129).
            auto at = [&](int i) -> XS {
                if (i < 0) return xsZero();
                const XS v = val[(size_t)i * 32 + lane];
                return splitNorm((double)v.m, v.e);
            };
            const XS p1 = at(L - 1), p2 = at(L - 2), p3 = at(L - 3);
            const double keepSingle = 1.0 - r.single;
            const double keepBoth = keepSingle - r.dbl;
            const XS trailingSingle = scaleScore(p2, keepSingle * 0.25);
            const XS trailingDouble = scaleScore(p3, keepBoth * 0.0625);
            const XS total = scalarAdd(scalarAdd(p1, trailingSingle), trailingDouble);
            const float nullLog = (total.m == 0.0f) ? -INFINITY : (float)(log2((double)total.m) + (double)total.e);
            double perBaseLog = -(double)nullLog / (double)L;
            if (!(perBaseLog < 120.0)) perBaseLog = 120.0;
            const double perBaseRaw = exp2(perBaseLog);
            const XS perBase = splitNorm(perBaseRaw, 0);
            baseAll[jw][0][lane] = perBase;
            baseAll[jw][1][lane] = splitNorm(1.0 / perBaseRaw, 0);
            if (on) {
                const XS quarter = splitNorm(0.25, 0), sixteenth = splitNorm(0.0625, 0);
                PairScales sc;
                sc.s1 = packScore(scalarMul(perBase, quarter));
                sc.s2 = packScore(scalarMul(scalarMul(perBase, perBase), sixteenth));
                sc.sC = packScore(scalarMul(scalarMul(perBase, perBase), perBase));
                sc.pad = 0.0f;
                scales[pi] = sc;
            }
        }
        pairSync();
        const XS perBase = baseAll[jw][0][lane], perBaseInv = baseAll[jw][1][lane];
        const int *len = lenAll[warp];
        float *const *dst = dstAll[warp];
        if (scaled) {
            if (suffixWarp ? seedScaled<true>(val, L, Lmax, powerScaled(perBase, L, Lmax), perBaseInv, stage, dst, len,
                                              job.count, lane)
                           : seedScaled<false>(val, L, Lmax, perBase, perBase, stage, dst, len, job.count, lane))
                continue;
            algebraPass(cd, L, Lmax, tab, keep, bg0, val, lane, r, suffixWarp);
        }
        if (suffixWarp) {
            // the suffix seeds' power starts at perBase^(L-1), one rounded product at a time
            XS running = pow2Score(0);
            for (int k = 1; k < Lmax; ++k) {
                const XS t = mulF(running, perBase);
                if (k < L) running = t;
            }
            seedPass<true>(val, L, Lmax, running, perBaseInv, stage, dst, len, job.count, lane);
        } else {
            seedPass<false>(val, L, Lmax, perBase, perBase, stage, dst, len, job.count, lane);
        }
    }
}

}  // namespace dmst
