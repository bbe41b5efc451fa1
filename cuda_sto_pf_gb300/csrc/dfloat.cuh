// dfloat.cuh — double-float arithmetic on the FP32 pipe.
//
// A value is the unevaluated sum hi + lo of two floats with |lo| <= ulp(hi)/2
// (about 48 significant bits).  Error-free transforms: Knuth's two-sum,
// Dekker's fast two-sum (|a| >= |b|) and the two-product through the fused
// multiply-add; the sums and products below follow the "sloppy" double-double
// forms of Hida, Li and Bailey (QD library paper, 2001), relative error a few
// units of 2^-48.  GB300 runs FP64 at 1/64 of the FP32 rate, so a per-cell
// evaluation that needs more than float precision is cheaper in this form
// than in double.
#pragma once

#include "dfexp.cuh"

struct dfl { float hi, lo; };

__device__ __forceinline__ dfl df_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ dfl df_fast_two_sum(float a, float b) {   // |a| >= |b| or a == 0
    const float s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ dfl df_two_prod(float a, float b) {
    const float p = a * b;
    return {p, fmaf(a, b, -p)};
}
__device__ __forceinline__ dfl df_add(dfl a, dfl b) {
    dfl s = df_two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return df_fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ dfl df_add_f(dfl a, float b) {
    dfl s = df_two_sum(a.hi, b);
    s.lo += a.lo;
    return df_fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ dfl df_mul(dfl a, dfl b) {
    dfl p = df_two_prod(a.hi, b.hi);
    p.lo = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, p.lo));
    return df_fast_two_sum(p.hi, p.lo);
}
__device__ __forceinline__ dfl df_mul_f(dfl a, float b) {
    dfl p = df_two_prod(a.hi, b);
    p.lo = fmaf(a.lo, b, p.lo);
    return df_fast_two_sum(p.hi, p.lo);
}
__device__ __forceinline__ dfl df_neg(dfl a) { return {-a.hi, -a.lo}; }
// 1 / d for d >= 1 (one Newton step from the float reciprocal: q0 + q0 (1 - d q0))
__device__ __forceinline__ dfl df_rcp(dfl d) {
    const float q0 = 1.0f / d.hi;
    float e = fmaf(-d.hi, q0, 1.0f);   // exact: q0 is the rounded quotient
    e = fmaf(-d.lo, q0, e);
    return df_fast_two_sum(q0, q0 * e);
}
__device__ __forceinline__ double df_to_double(dfl a) { return (double)a.hi + (double)a.lo; }
__device__ __forceinline__ dfl df_from_double(double v) {
    const float hi = (float)v;
    return {hi, (float)(v - (double)hi)};
}

// ---------------------------------------------------------------------------
// Values that end as floats: the float that the same expression in FP64 rounds
// to, found in double-float arithmetic wherever it decides it (Ziv, "Fast
// Evaluation of Elementary Mathematical Functions with Correctly Rounded Last
// Bit", ACM TOMS 17, 1991).  The double-float value is f + c; if everything
// within 2^-40 of it rounds to one float, so does the double value, which lies
// within 2^-42.  The rest, one value in some 2^15, and what leaves the range that
// this holds for, is the caller's to compute in FP64.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool df_rounds(float f, float c, float *out) {
    const float err = fabsf(f) * 0x1p-40f;
    const float lo = f + (c - err), hi = f + (c + err);
    *out = lo;
    return lo == hi && fabsf(f) > 0x1p-80f && fabsf(f) < 0x1p100f;
}
// float(a b) for |a b| in (2^-80, 2^100)
__device__ __forceinline__ bool df_round_product(dfl a, dfl b, float *out) {
    const dfl p = df_mul(a, b);
    return df_rounds(p.hi, p.lo, out);
}
// float(num / (1 + m k2)) for 1 + m k2 in [1/2, 2^60): one correction of the
// float quotient
__device__ __forceinline__ bool df_round_damped(dfl num, dfl m, dfl k2, float *out) {
    const dfl den = df_add_f(df_mul(m, k2), 1.0f);
    const float q = 1.0f / den.hi, f = num.hi * q;
    const float e = fmaf(-f, den.hi, num.hi) + fmaf(-f, den.lo, num.lo);
    return df_rounds(f, e * q, out) && den.hi >= 0.5f && den.hi < 0x1p60f && fabsf(m.hi) < 0x1p60f && k2.hi < 0x1p60f;
}

// ---------------------------------------------------------------------------
// A sum of floats, or of their exact products, in more than a double's 53 bits
// on the FP32 pipe: h + m + l, where m holds the rounding errors of h and l
// those of m (cascaded compensated summation, Ogita, Rump and Oishi, 2005: as
// if summed with 72 bits), and in x what float arithmetic has no room for (sums
// that could overflow, products whose error term would underflow, infinities and
// NaN), in FP64 as a plain double sum has it.
// ---------------------------------------------------------------------------
struct fsum { float h, m, l; double x; };

__device__ __forceinline__ fsum fs_zero() { return {0.f, 0.f, 0.f, 0.0}; }
// s += v at the level of m (an error term of what h takes)
__device__ __forceinline__ void fs_add_low(fsum &s, float v) {
    const dfl u = df_two_sum(s.m, v);
    s.m = u.hi;
    s.l += u.lo;
}
__device__ __forceinline__ void fs_add_in_range(fsum &s, float v) {
    const dfl t = df_two_sum(s.h, v);
    s.h = t.hi;
    fs_add_low(s, t.lo);
}
__device__ __forceinline__ void fs_add(fsum &s, float v) {
    if (fabsf(v) < 0x1p96f) fs_add_in_range(s, v);   // 2^31 of them stay below a float's range
    else s.x += (double)v;
}
// s += v^2: the two-product is exact for 2^-46 < |v| < 2^48 and for 0
__device__ __forceinline__ void fs_add_square(fsum &s, float v) {
    const float a = fabsf(v);
    if ((a > 0x1p-46f && a < 0x1p48f) || a == 0.f) {
        const dfl p = df_two_prod(v, v);
        fs_add_in_range(s, p.hi);
        fs_add_low(s, p.lo);
    } else {
        s.x += (double)v * (double)v;
    }
}
// s += (p - q)^2, where the difference is a float (it is for values within a factor
// of two), and in FP64 where it is not
__device__ __forceinline__ void fs_add_square_diff(fsum &s, float p, float q) {
    const dfl d = df_two_sum(p, -q);
    if (d.lo == 0.f) fs_add_square(s, d.hi);
    else s.x += ((double)p - (double)q) * ((double)p - (double)q);
}
// s += a d for a difference d = df_two_sum(p, -q), if it is in the range that the
// exact products have
__device__ __forceinline__ bool fs_add_product(fsum &s, float a, dfl d) {
    const float u = fabsf(a), v = fabsf(d.hi);
    if (!((u > 0x1p-46f && u < 0x1p48f) || u == 0.f) || !((v > 0x1p-46f && v < 0x1p48f) || v == 0.f)) return false;
    const dfl p = df_two_prod(a, d.hi), r = df_two_prod(a, d.lo);
    fs_add_in_range(s, p.hi);
    fs_add_low(s, p.lo);
    fs_add_low(s, r.hi);
    s.l += r.lo;
    return true;
}
__device__ __forceinline__ void fs_merge(fsum &s, const fsum &b) {
    fs_add_in_range(s, b.h);
    fs_add_low(s, b.m);
    s.l += b.l;
    if (__double_as_longlong(b.x) != 0) s.x += b.x;   // (a branch, not an FP64 addition)
}
__device__ __forceinline__ fsum fs_shfl_down(const fsum &s, int o) {
    const unsigned all = 0xffffffffu;
    return {__shfl_down_sync(all, s.h, o), __shfl_down_sync(all, s.m, o), __shfl_down_sync(all, s.l, o),
            __shfl_down_sync(all, s.x, o)};
}
__device__ __forceinline__ double fs_to_double(const fsum &s) {
    return s.x + ((double)s.h + ((double)s.m + (double)s.l));
}

// e^w for -40 <= w <= 0 by Tang's table-driven method (ACM TOMS 15, 1989):
// w = N ln2/64 + r (N = 64 k + j, |r| <= ln2/128),
// e^r = 1 + r + r^2/2 + (r^3/6 + r^4/24 + r^5/120) with the bracket in
// float (below 2.7e-8, so its rounding is under 2^-48 of the result), times
// 2^(j/64) from the double-float table, times 2^k (exact).
// tab: dfexp::kExp2Tab staged in shared memory
__device__ __forceinline__ dfl df_exp_neg(dfl w, const float2 *tab) {
    // N = nearest integer to w.hi * 64/ln2 (-3694 .. 0) by the 1.5 * 2^23
    // shift: its float bits hold N, so no float <-> int conversion is issued
    const float tN = fmaf(w.hi, dfexp::kInvL64, 12582912.0f);
    const float fN = tN - 12582912.0f;
    const int N = __float_as_int(tN) - 0x4B400000;
    // w.hi - N C1 is exact (N C1 has 24 bits and is within a factor 2 of w.hi)
    dfl r = df_two_sum(fmaf(-fN, dfexp::kC1, w.hi), w.lo);
    r = df_add(r, df_neg(df_two_prod(fN, dfexp::kC2)));
    r = df_add_f(r, -fN * dfexp::kC3);
    const float rh = r.hi;
    const float tail = rh * rh * rh * (1.0f / 6.0f + rh * (1.0f / 24.0f + rh * (1.0f / 120.0f)));
    dfl q = df_two_prod(rh, rh);   // r^2 / 2 with the lo part of r
    q.lo = fmaf(2.0f * rh, r.lo, q.lo);
    q.hi *= 0.5f;
    q.lo *= 0.5f;
    dfl e = df_add_f(q, tail);
    e = df_add(e, r);
    e = df_add_f(e, 1.0f);
    const int j = N & 63, k = (N - j) / 64;   // N = 64 k + j, 0 <= j < 64, -58 <= k <= 0
    const float2 t = tab[j];
    e = df_mul(e, dfl{t.x, t.y});
    const float s = __int_as_float((127 + k) << 23);   // 2^k, a normal float
    return {e.hi * s, e.lo * s};
}

// sigmoid(z) = 1 / (1 + e^-z) of a double-float z; beyond |z| = 40 the
// float sigmoid (the double-float correction is below 4e-18 there)
__device__ __forceinline__ dfl df_sigmoid(dfl z, const float2 *tab) {
    if (!(fabsf(z.hi) <= 40.0f)) {
        const float zf = z.hi;
        const float s = zf >= 0.0f ? 1.0f / (1.0f + __expf(-zf)) : __expf(zf) / (1.0f + __expf(zf));
        return {s, 0.0f};
    }
    const bool pos = z.hi >= 0.0f;
    const dfl E = df_exp_neg(pos ? df_neg(z) : z, tab);   // e^-|z| <= 1
    const dfl r = df_rcp(df_add_f(E, 1.0f));
    return pos ? r : df_mul(E, r);
}
