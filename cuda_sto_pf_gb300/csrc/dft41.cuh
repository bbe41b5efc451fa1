// dft41.cuh — the 41-point DFT of one thread, as Rader's cyclic convolution
// split by the Chinese remainder theorem (Rader 1968; Nussbaumer, "Fast
// Fourier Transform and Convolution Algorithms", 1982).
//
// 6 generates the residues mod 41: n = 6^s, q = 6^t.  With a_s = y_(6^s) +
// y_(-6^s) and b_s = y_(6^s) - y_(-6^s) (6^20 = -1),
//   X_(6^t)  = y_0 + C_t + DIR i S_t,   X_(-6^t) = y_0 + C_t - DIR i S_t
//   C_t = sum_(s mod 20) a_s cos(2 pi 6^(s+t) / 41)                 cyclic, Z_20
//   S_t = sum_(s < 20)   b_s sin(2 pi 6^(s+t) / 41)   sign-cyclic (s + 20 -> -)
// Z_20 = Z_4 x Z_5 and Z_40 = Z_8 x Z_5 turn both into 5-point cyclic
// correlations of 4-point transforms over the other index: C into two real
// ones and a complex one (the factors z - 1, z + 1, z^2 + 1 of z^4 - 1), S
// into two complex ones (the roots e^(i pi / 4), e^(3 i pi / 4) of z^4 + 1).
// That is 350 multiply-adds for a real line against 800 of the direct
// symmetric form (20 x 20 cosines and as many sines), and every output of
// one beta (the index mod 5) needs eight accumulators only.
//
// Each operation acts on the real and the imaginary part of a value with
// the same constant: packed f32x2 arithmetic (two roundings to nearest per
// instruction, the same values as the scalar instructions).
#pragma once

#include "common.cuh"
#include "f32x2.cuh"
#include "rader41.cuh"

namespace d41 {

__host__ __device__ constexpr int pow6(int s) {
    int p = 1;
    for (int i = 0; i < s; ++i) p = (p * 6) % 41;
    return p;
}
// the s with s = a (mod ma), s = b (mod 5)
__host__ __device__ constexpr int crt(int a, int ma, int b) {
    for (int s = 0; s < 5 * ma; ++s)
        if (s % ma == a && s % 5 == b) return s;
    return 0;
}
__host__ __device__ constexpr double cab(int a, int b) { return dft41_cos(pow6(crt(a, 4, b))); }
__host__ __device__ constexpr double hab(int a, int b) { return dft41_sin(pow6(crt(a, 8, b))); }
constexpr double R2 = 0.70710678118654752440084436210485;   // cos(pi / 4)

// the constants of one b: C's factors (sums over alpha, scaled for the
// 4-point inverse), then F = sum_v h_v w^v / 2 at the two roots w
enum { CPP, CPM, H0, H1, F1R, F1I, F3R, F3I, NCONST };
__host__ __device__ constexpr double cval(int which, int b) {
    const double c0 = cab(0, b), c1 = cab(1, b), c2 = cab(2, b), c3 = cab(3, b);
    const double h0 = hab(0, b), h1 = hab(1, b), h2 = hab(2, b), h3 = hab(3, b);
    return which == CPP   ? 0.25 * (c0 + c1 + c2 + c3)
           : which == CPM ? 0.25 * (c0 - c1 + c2 - c3)
           : which == H0  ? 0.5 * (c0 - c2)
           : which == H1  ? 0.5 * (c1 - c3)
           : which == F1R ? 0.5 * (h0 + R2 * (h1 - h3))
           : which == F1I ? 0.5 * (h2 + R2 * (h1 + h3))
           : which == F3R ? 0.5 * (h0 - R2 * (h1 - h3))
                          : 0.5 * (-h2 + R2 * (h1 + h3));
}

using namespace f2x;
template <int W, int B, bool NEG = false> __device__ __forceinline__ P kc() {
    constexpr float k = (float)(NEG ? -cval(W, B) : cval(W, B));
    return both(k);
}
template <int W, int B, bool NEG = false> __device__ __forceinline__ P mad(P a, P c) { return fma(a, kc<W, B, NEG>(), c); }
template <int W, int B> __device__ __forceinline__ P mulc(P a) { return mul(a, kc<W, B>()); }
template <bool NEG> __device__ __forceinline__ P madr(P a, P c) { return fma(a, both(NEG ? -(float)R2 : (float)R2), c); }
__device__ __forceinline__ P mulr(P a) { return mul(a, both((float)R2)); }

// the 41 inputs after the first, transformed over the 4-point index: per b
// mod 5 the inputs of the five correlations
struct In { P y0, pp[5], pm[5], m0[5], m1[5], xr[5], xi[5], zr[5], zi[5]; };

template <int B, class F> __device__ __forceinline__ void load_b(In &v, F &&get) {
    // the four pairs (n, 41 - n) with this index mod 5: s over Z_20 for the
    // sums, over Z_40 (where 41 - n is n's s + 20) for the differences
    P a[4], b[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const int n = pow6(crt(l, 4, B));
        a[l] = add(pk(get(n)), pk(get(41 - n)));
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const int n = pow6(crt(l, 8, B));
        b[l] = sub(pk(get(n)), pk(get(41 - n)));
    }
    const P e = add(a[0], a[2]), o = add(a[1], a[3]);
    v.pp[B] = add(e, o);
    v.pm[B] = sub(e, o);
    v.m0[B] = sub(a[0], a[2]);
    v.m1[B] = sub(a[1], a[3]);
    const P d = sub(b[1], b[3]), s = add(b[1], b[3]);
    v.xr[B] = madr<false>(d, b[0]);
    v.zr[B] = madr<true>(d, b[0]);
    v.xi[B] = madr<false>(s, b[2]);
    v.zi[B] = madr<true>(s, b[2]);
}

template <int T, int K> struct Acc {
    static __device__ __forceinline__ void go(const In &v, P &pp, P &pm, P &a0, P &a1, P &r1, P &i1, P &r3, P &i3) {
        constexpr int U = (K + T) % 5;
        pp = mad<CPP, U>(v.pp[K], K == 0 ? v.y0 : pp);
        if (K == 0) {
            pm = mulc<CPM, U>(v.pm[K]);
            a0 = mulc<H0, U>(v.m0[K]);
            a1 = mulc<H1, U>(v.m0[K]);
            r1 = mulc<F1R, U>(v.xr[K]);
            i1 = mulc<F1I, U>(v.xr[K]);
            r3 = mulc<F3R, U>(v.zr[K]);
            i3 = mulc<F3I, U>(v.zr[K]);
        } else {
            pm = mad<CPM, U>(v.pm[K], pm);
            a0 = mad<H0, U>(v.m0[K], a0);
            a1 = mad<H1, U>(v.m0[K], a1);
            r1 = mad<F1R, U>(v.xr[K], r1);
            i1 = mad<F1I, U>(v.xr[K], i1);
            r3 = mad<F3R, U>(v.zr[K], r3);
            i3 = mad<F3I, U>(v.zr[K], i3);
        }
        a0 = mad<H1, U>(v.m1[K], a0);
        a1 = mad<H0, U, true>(v.m1[K], a1);
        r1 = mad<F1I, U>(v.xi[K], r1);
        i1 = mad<F1R, U, true>(v.xi[K], i1);
        r3 = mad<F3I, U, true>(v.zi[K], r3);
        i3 = mad<F3R, U>(v.zi[K], i3);
        if constexpr (K < 4) Acc<T, K + 1>::go(v, pp, pm, a0, a1, r1, i1, r3, i3);
    }
};

template <int DIR, int T, int L, class F> __device__ __forceinline__ void emit(P c_, P s_, F &&put) {
    constexpr int q = pow6(crt(L, 8, T));
    const float2 c = un(c_), s = un(s_);
    // DIR i S with i S = (-S.y, S.x)
    const float dx = DIR < 0 ? s.y : -s.y, dy = DIR < 0 ? -s.x : s.x;
    put(q, make_float2(c.x + dx, c.y + dy));
    put(41 - q, make_float2(c.x - dx, c.y - dy));
}

template <int DIR, int T, class F> __device__ __forceinline__ void out_t(const In &v, F &&put) {
    P pp, pm, a0, a1, r1, i1, r3, i3;
    Acc<T, 0>::go(v, pp, pm, a0, a1, r1, i1, r3, i3);
    const P e = add(pp, pm), o = sub(pp, pm);
    const P u = sub(r1, r3), w = add(i1, i3);
    emit<DIR, T, 0>(add(e, a0), add(r1, r3), put);
    emit<DIR, T, 2>(sub(e, a0), sub(i1, i3), put);
    emit<DIR, T, 1>(add(o, a1), mulr(add(u, w)), put);
    emit<DIR, T, 3>(sub(o, a1), mulr(sub(w, u)), put);
}

// get(n), n = 0..40: the inputs; put(q, X_q): the outputs, X_0 first
template <class F> __device__ __forceinline__ void load(In &v, F &&get) {
    v.y0 = pk(get(0));
    load_b<0>(v, get); load_b<1>(v, get); load_b<2>(v, get); load_b<3>(v, get); load_b<4>(v, get);
}
template <int DIR, class F> __device__ __forceinline__ void store(const In &v, F &&put) {
    put(0, un(add(add(v.y0, v.pp[0]), add(add(v.pp[1], v.pp[2]), add(v.pp[3], v.pp[4])))));
    out_t<DIR, 0>(v, put); out_t<DIR, 1>(v, put); out_t<DIR, 2>(v, put); out_t<DIR, 3>(v, put); out_t<DIR, 4>(v, put);
}

}  // namespace d41
