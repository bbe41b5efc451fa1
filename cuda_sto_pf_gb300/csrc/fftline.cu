// fftline.cu — the line transforms of the generic engine (fft.cuh): in-place
// mixed-radix stages in shared memory.  Compiled once for each precision and
// direction (PFGB_LINE_T, PFGB_LINE_DIR), as relocatable device code that the
// pass kernels call.
#include "fft.cuh"

// cos and sin of 2 pi i / N at compile time (the Taylor series on an octant,
// exact to the last bits of a double)
constexpr double ct_series(double x, bool sine) {
    double t = sine ? x : 1.0, sum = t;
    for (int k = sine ? 3 : 2; k < 30; k += 2) {
        t *= -x * x / ((k - 1) * k);
        sum += t;
    }
    return sum;
}
template <int N>
struct Roots {
    double c[N] = {}, s[N] = {};
    constexpr Roots() {
        for (int i = 0; i < N; ++i) {
            // eighths of a turn: 8 i = a N + r, the angle folded to r or N - r
            const int a = 8 * i / N, r = 8 * i % N;
            const double x = PFGB_PI / 4.0 * (a % 2 ? N - r : r) / N;
            const double u = ct_series(x, false), v = ct_series(x, true);
            const bool sw = a % 4 == 1 || a % 4 == 2;   // cos and sin exchanged
            c[i] = (a >= 2 && a <= 5 ? -1.0 : 1.0) * (sw ? v : u);
            s[i] = (a >= 4 ? -1.0 : 1.0) * (sw ? u : v);
        }
    }
};
template <int N>
__host__ __device__ constexpr double root_c(int i) {
    constexpr Roots<N> t;
    return t.c[i % N];
}
template <int N>
__host__ __device__ constexpr double root_s(int i) {
    constexpr Roots<N> t;
    return t.s[i % N];
}

// prime radices 7, 11 and 13 by the symmetric form: a_j = v_j + v_(R-j), b_j =
// v_j - v_(R-j); X_k = v_0 + sum a_j cos(2 pi j k / R) + DIR i sum b_j sin(..)
template <typename T, int DIR, int R>
__device__ __forceinline__ void bfly_odd(cplx_t<T> *v) {
    using T2 = cplx_t<T>;
    constexpr int H = R / 2;
    T2 a[H], b[H], s = v[0];
#pragma unroll
    for (int j = 1; j <= H; ++j) {
        a[j - 1] = padd(v[j], v[R - j]);
        b[j - 1] = psub(v[j], v[R - j]);
        s = padd(s, a[j - 1]);
    }
    const T2 v0 = v[0];
    v[0] = s;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        T2 c = v0, d = mk2<T2>(T(0), T(0));
#pragma unroll
        for (int j = 1; j <= H; ++j) {
            const T co = T(root_c<R>(j * k)), si = T(root_s<R>(j * k));
            c = mk2<T2>(c.x + a[j - 1].x * co, c.y + a[j - 1].y * co);
            d = mk2<T2>(d.x + b[j - 1].x * si, d.y + b[j - 1].y * si);
        }
        const T2 e = rot_mi<DIR>(d);   // DIR i d
        v[k] = padd(c, e);
        v[R - k] = psub(c, e);
    }
}

template <typename T, int DIR, int R> __device__ __forceinline__ void bfly(cplx_t<T> *v);
// composite radices R = P Q: Q-point DFTs over stride P, the twiddles
// W_R^(p q) and P-point DFTs
template <typename T, int DIR, int P, int Q>
__device__ __forceinline__ void bfly_pq(cplx_t<T> *v) {
    using T2 = cplx_t<T>;
    T2 w[P][Q];
#pragma unroll
    for (int p = 0; p < P; ++p) {
#pragma unroll
        for (int q = 0; q < Q; ++q) w[p][q] = v[p + P * q];
        bfly<T, DIR, Q>(w[p]);
    }
    if constexpr (P == 2 && sizeof(T) == 4) {   // the twiddles' products fused into the last sums
        v[0] = padd(w[0][0], w[1][0]);
        v[Q] = psub(w[0][0], w[1][0]);
#pragma unroll
        for (int q = 1; q < Q; ++q) {
            const T co = T(root_c<P * Q>(q)), si = T(root_s<P * Q>(q));
            const T2 x = w[1][q], r = rot_mi<DIR>(x);
            v[q] = pmad(x, co, pmad(r, si, w[0][q]));
            v[q + Q] = pmad(x, -co, pmad(r, -si, w[0][q]));
        }
        return;
    }
#pragma unroll
    for (int p = 1; p < P; ++p)
#pragma unroll
        for (int q = 1; q < Q; ++q) {
            const T co = T(root_c<P * Q>(p * q)), si = T(root_s<P * Q>(p * q));
            const T sg = DIR < 0 ? -si : si;
            const T2 x = w[p][q];
            w[p][q] = mk2<T2>(x.x * co - x.y * sg, x.x * sg + x.y * co);
        }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        T2 u[P];
#pragma unroll
        for (int p = 0; p < P; ++p) u[p] = w[p][q];
        bfly<T, DIR, P>(u);
#pragma unroll
        for (int p = 0; p < P; ++p) v[q + Q * p] = u[p];
    }
}

template <typename T, int DIR, int R>
__device__ __forceinline__ void bfly(cplx_t<T> *v) {
    if constexpr (R == 2) bfly2<T, DIR>(v);
    else if constexpr (R == 3) bfly3<T, DIR>(v);
    else if constexpr (R == 4) bfly4<T, DIR>(v);
    else if constexpr (R == 5) bfly5<T, DIR>(v);
    else if constexpr (R == 6) bfly6<T, DIR>(v);
    else if constexpr (R == 8) bfly8<T, DIR>(v);
    else if constexpr (R == 9) bfly_pq<T, DIR, 3, 3>(v);
    else if constexpr (R == 10) bfly_pq<T, DIR, 2, 5>(v);
    else if constexpr (R == 12) bfly_pq<T, DIR, 3, 4>(v);
    else if constexpr (R == 14) bfly_pq<T, DIR, 2, 7>(v);
    else if constexpr (R == 15) bfly_pq<T, DIR, 3, 5>(v);
    else if constexpr (R == 16) bfly_pq<T, DIR, 4, 4>(v);
    else bfly_odd<T, DIR, R>(v);
}

__device__ __forceinline__ float2 lds2(uint32_t a, float) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double2 lds2(uint32_t a, double) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts2(uint32_t a, float2 v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sts2(uint32_t a, double2 v) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}

// a += s, each time anew: as a + r s the offsets r s would be kept in registers
// over the loop of a stage, and a stage saves to the stack what it uses of them
__device__ __forceinline__ void advance(uint32_t &a, uint32_t s) { asm volatile("add.u32 %0, %0, %1;" : "+r"(a) : "r"(s)); }

// natural position of output r = 0 of block b of the last stage: b's digits
// (k_1 most significant) in the reverse order of significance
__device__ __forceinline__ int reversed_block(const AxisPlan &p, int b) {
    int out = 0;
    for (int s = p.nst - 2; s >= 0; --s) {
        const int R = p.st[s].R, q = (int)p.st[s].fR.div((unsigned)b);
        out = out * R + (b - q * R);
        b = q;
    }
    return out;
}

template <typename T, int DIR, int R>
__device__ __noinline__ void stage_mid(LineTile t, int nb, int B, int m, int twst, FastDiv fm) {
    using T2 = cplx_t<T>;
    const int L = (int)t.fL.d, items = L * nb, step = m * t.PS;
#pragma unroll 1
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        const int j = (int)t.fL.div((unsigned)it), l = it - j * L;
        const int b = (int)fm.div((unsigned)j), jp = j - b * m;
        const uint32_t a0 = t.buf + (uint32_t)((b * B + jp) * t.PS + l * t.LS);
        uint32_t a = a0;
        T2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { v[r] = lds2(a, T(0)); advance(a, step); }
        bfly<T, DIR, R>(v);
        const uint32_t wst = (uint32_t)(jp * twst) * (uint32_t)sizeof(T2);
        uint32_t wa = t.tw;
#pragma unroll
        for (int r = 1; r < R; ++r) { advance(wa, wst); v[r] = twmul<DIR>(v[r], lds2(wa, T(0))); }
        a = a0;
#pragma unroll
        for (int r = 0; r < R; ++r) { sts2(a, v[r]); advance(a, step); }
    }
}

// the last stage: a chunk of lines at a time, one butterfly per thread, whose
// points are all in registers before the block writes them back.  A block has
// a thread for every butterfly of a line (pfgb_make_plan, pfgb_line_threads),
// so that a chunk holds at least one line.
template <typename T, int DIR, int R>
__device__ __noinline__ void stage_last(LineTile t, const AxisPlan *plan, int nb) {
    using T2 = cplx_t<T>;
    const AxisPlan &p = *plan;
    const int L = (int)t.fL.d, Lc = min(L, (int)blockDim.x / nb), ost = nb * t.PS;
    // this thread's block j of line l of every chunk
    const int j = (int)threadIdx.x / Lc, l = (int)threadIdx.x - j * Lc;
    const uint32_t in = t.buf + (uint32_t)(j * R * t.PS), out = t.buf + (uint32_t)(reversed_block(p, j) * t.PS);
#pragma unroll 1
    for (int l0 = 0; l0 < L; l0 += Lc) {
        const bool act = j < nb && l0 + l < L;
        const uint32_t lo = (uint32_t)((l0 + l) * t.LS);
        T2 v[R];
        if (act) {
            uint32_t a = in + lo;
#pragma unroll
            for (int r = 0; r < R; ++r) { v[r] = lds2(a, T(0)); advance(a, t.PS); }
            bfly<T, DIR, R>(v);
        }
        __syncthreads();
        if (act) {
            uint32_t a = out + lo;
#pragma unroll
            for (int r = 0; r < R; ++r) { sts2(a, v[r]); advance(a, ost); }
        }
    }
}

// any other prime radix: each output is a direct sum over its R inputs,
// out_k = sum_r x_r W_n^(twst k (r m + j')) (the DFT and its twiddle in one
// exponent); eight outputs per thread wait in registers for the block
template <typename T, int DIR>
__device__ __noinline__ void stage_direct(LineTile t, const AxisPlan *plan, int s) {
    using T2 = cplx_t<T>;
    constexpr int H = PFGB_DIRECT_SUMS;
    const AxisPlan &p = *plan;
    const int n = p.n, R = p.st[s].R, B = p.st[s].B, m = p.st[s].m, twst = n / B;
    const FastDiv fm = p.st[s].fm;
    const bool last = s == p.nst - 1;
    const int L = (int)t.fL.d, Lc = min(L, (int)blockDim.x * H / n), nb = n / R;
#pragma unroll 1
    for (int l0 = 0; l0 < L; l0 += Lc) {
        const int lc = min(Lc, L - l0), items = lc * n;
        T2 acc[H];
        uint32_t o[H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int it = threadIdx.x + h * blockDim.x;
            if (it < items) {
                const int q = it / lc, l = l0 + it - q * lc;
                const int b = q / B, k = (int)fm.div((unsigned)(q - b * B)), jp = q - b * B - k * m;
                const uint32_t base = t.buf + (uint32_t)(l * t.LS);
                const uint32_t a = base + (uint32_t)((b * B + jp) * t.PS);
                o[h] = base + (uint32_t)((last ? reversed_block(p, b) + k * nb : q) * t.PS);
                int idx = k * jp * twst;             // < n
                const int step = k * m * twst;       // < n
                T ar = 0, ai = 0;
                for (int r = 0; r < R; ++r) {
                    const T2 x = lds2(a + r * m * t.PS, T(0)), w = lds2(t.tw + idx * (int)sizeof(T2), T(0));
                    if (DIR < 0) { ar += x.x * w.x - x.y * w.y; ai += x.x * w.y + x.y * w.x; }
                    else { ar += x.x * w.x + x.y * w.y; ai += x.y * w.x - x.x * w.y; }
                    idx += step;
                    if (idx >= n) idx -= n;
                }
                acc[h] = mk2<T2>(ar, ai);
            }
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < H; ++h)
            if ((int)(threadIdx.x + h * blockDim.x) < items) sts2(o[h], acc[h]);
    }
}

// ---------------------------------------------------------------------------
// Radix-41 stage (always a line's first) by Rader's algorithm, 8 lanes per
// 41-point DFT.
//   X_0 = sum x ;  X_{7^q} = x_0 + (a (*) b)_q,  a_p = x_{6^p}  (mod 41)
// The length-40 cyclic convolution is IFFT40(FFT40(a) . B) with
// B = FFT40(b)/40 (rader41.cuh).  FFT40 = 5 x 8: lane t (0..7) owns
// a[t + 8m], m = 0..4, does the 5-point DFTs in registers, the W40^{t k1}
// twiddles, and the 8-point DFTs run across the 8 lanes with shuffles
// (decimation in frequency forward -> bit-reversed lanes, decimation in time
// inverse -> natural lanes).  Index maps: 6^(t+8m) = 6^t 10^m, 7^(t+8m) =
// 7^t 37^m (mod 41).
// ---------------------------------------------------------------------------
template <typename T> struct RaderTab;
template <> struct RaderTab<float> {
    static __device__ __forceinline__ float2 B(int dir, int k) { return dir < 0 ? c_rader41_BF_f[k] : c_rader41_BI_f[k]; }
};
template <> struct RaderTab<double> {
    static __device__ __forceinline__ double2 B(int dir, int k) { return dir < 0 ? c_rader41_BF_d[k] : c_rader41_BI_d[k]; }
};

template <typename T2>
__device__ __forceinline__ T2 shfl_x(T2 v, int m, unsigned mask) {
    v.x = __shfl_xor_sync(mask, v.x, m, 8);
    v.y = __shfl_xor_sync(mask, v.y, m, 8);
    return v;
}

template <typename T, int DIR>
__device__ __noinline__ void stage_rader41(LineTile tl, int nb) {
    using T2 = cplx_t<T>;
    const int nl = (int)tl.fL.d;
    const int t = threadIdx.x & 7;
    const int group = threadIdx.x >> 3, ngroups = blockDim.x >> 3;
    const unsigned gmask = 0xffu << (threadIdx.x & 24);
    const int brt = ((t & 1) << 2) | (t & 2) | ((t & 4) >> 2);
    // per-lane constants: W40^{t k1}, B[k1 + 5 br(t)], butterfly signs/twiddles,
    // and the shared-memory offsets of the lane's 5 inputs and 5 outputs
    T2 W[5], Bk[5];
#pragma unroll
    for (int k1 = 0; k1 < 5; ++k1) {
        T sn, cs;
        if constexpr (sizeof(T) == 4) sincospif(-2.0f * (float)(t * k1) / 40.0f, &sn, &cs);
        else sincospi(-2.0 * (double)(t * k1) / 40.0, &sn, &cs);
        W[k1] = mk2<T2>(cs, sn);
        Bk[k1] = RaderTab<T>::B(DIR, k1 + 5 * brt);
    }
    const T r = T(0.70710678118654752440084436210485);
    const int p4 = t & 3, p2 = t & 1;
    // forward twiddles of the lane's DIF butterflies (W8^{p4}, W4^{p2}); the
    // lower lane of a pair uses 1 and sign +1, the upper one f and sign -1
    const T2 one = mk2<T2>(T(1), T(0));
    const T2 f4 = p4 == 0 ? one : p4 == 1 ? mk2<T2>(r, -r) : p4 == 2 ? mk2<T2>(T(0), T(-1)) : mk2<T2>(-r, -r);
    const T2 f2 = p2 == 0 ? one : mk2<T2>(T(0), T(-1));
    const T s4 = (t & 4) ? T(-1) : T(1), s2 = (t & 2) ? T(-1) : T(1), s1 = (t & 1) ? T(-1) : T(1);
    const T2 w4 = (t & 4) ? f4 : one, w2 = (t & 2) ? f2 : one;
    // inverse (DIT) twiddles W8^{+p4}, W4^{+p2} applied by the upper lane
    const T2 c4 = mk2<T2>(f4.x, -f4.y), c2 = mk2<T2>(f2.x, -f2.y);
    int inoff[5], oidx[5];
    {
        int n = 1, o = 1;
        for (int i = 0; i < t; ++i) { n = (n * 6) % 41; o = (o * 7) % 41; }
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            inoff[q] = n * nb * tl.PS;
            oidx[q] = o;
            n = (n * 10) % 41;
            o = (o * 37) % 41;
        }
    }
    const int items = nl * nb;
    for (int it = group; it < items; it += ngroups) {
        const int j = (int)tl.fL.div((unsigned)it), l = it - j * nl;
        const uint32_t sb = tl.buf + (uint32_t)(j * tl.PS + l * tl.LS);
        T2 v[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) v[q] = lds2(sb + inoff[q], T(0));
        const T2 x0 = lds2(sb, T(0));
        // X_0 = x_0 + sum over the 40 permuted inputs
        T2 s = padd(padd(padd(v[0], v[1]), padd(v[2], v[3])), v[4]);
        s = padd(s, shfl_x(s, 1, gmask));
        s = padd(s, shfl_x(s, 2, gmask));
        s = padd(s, shfl_x(s, 4, gmask));
        // forward FFT40 of a: in-lane DFT5, twiddle, cross-lane DFT8 (DIF)
        bfly5<T, -1>(v);
#pragma unroll
        for (int q = 1; q < 5; ++q) v[q] = cmul(v[q], W[q]);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            // DIF: lower a + b, upper (a - b) w  ==  (partner + sign * own) * w_lane
            T2 u = shfl_x(v[q], 4, gmask);
            v[q] = cmul(mk2<T2>(u.x + s4 * v[q].x, u.y + s4 * v[q].y), w4);
            u = shfl_x(v[q], 2, gmask);
            v[q] = cmul(mk2<T2>(u.x + s2 * v[q].x, u.y + s2 * v[q].y), w2);
            u = shfl_x(v[q], 1, gmask);
            v[q] = mk2<T2>(u.x + s1 * v[q].x, u.y + s1 * v[q].y);
            v[q] = cmul(v[q], Bk[q]);
            // inverse DIT (bit-reversed in, natural out): the upper lane sends
            // w b; lower: a + (w b), upper: a - (w b)
            T2 sv = v[q];                                  // span 1: w = 1
            u = shfl_x(sv, 1, gmask);
            v[q] = (t & 1) ? psub(u, sv) : padd(v[q], u);
            sv = (t & 2) ? cmul(v[q], c2) : v[q];
            u = shfl_x(sv, 2, gmask);
            v[q] = (t & 2) ? psub(u, sv) : padd(v[q], u);
            sv = (t & 4) ? cmul(v[q], c4) : v[q];
            u = shfl_x(sv, 4, gmask);
            v[q] = (t & 4) ? psub(u, sv) : padd(v[q], u);
        }
#pragma unroll
        for (int q = 1; q < 5; ++q) v[q] = cmulconj(v[q], W[q]);
        bfly5<T, +1>(v);
        // outputs X[7^(t+8m)] = x0 + c[t+8m], twiddled, to the same places (the
        // shuffles above come after every lane's reads)
#pragma unroll
        for (int q = 0; q < 5; ++q)
            sts2(sb + (uint32_t)(oidx[q] * nb * tl.PS),
                 twmul<DIR>(padd(x0, v[q]), lds2(tl.tw + oidx[q] * j * (int)sizeof(T2), T(0))));
        if (t == 0) sts2(sb, padd(x0, s));
    }
}

// the stages of a plan one after another; ends with __syncthreads()
template <typename T, int DIR>
__device__ __forceinline__ void run_stages(const LineTile &t, const AxisPlan &p) {
    for (int s = 0; s < p.nst; ++s) {
        const int R = p.st[s].R, B = p.st[s].B, m = p.st[s].m, nb = p.n / R, twst = p.n / B;
        const FastDiv fm = p.st[s].fm;
        if (p.st[s].kind == 1) stage_rader41<T, DIR>(t, nb);
        else if (p.st[s].kind == 2) stage_direct<T, DIR>(t, &p, s);
        else if (s < p.nst - 1) {
            switch (R) {
#define PFGB_R(N) case N: stage_mid<T, DIR, N>(t, nb, B, m, twst, fm); break;
                PFGB_R(2) PFGB_R(3) PFGB_R(4) PFGB_R(5) PFGB_R(6) PFGB_R(7) PFGB_R(8) PFGB_R(9) PFGB_R(10) PFGB_R(11)
                PFGB_R(12) PFGB_R(13) PFGB_R(14) PFGB_R(15) PFGB_R(16)
#undef PFGB_R
            }
        } else {
            switch (R) {
#define PFGB_R(N) case N: stage_last<T, DIR, N>(t, &p, nb); break;
                PFGB_R(2) PFGB_R(3) PFGB_R(4) PFGB_R(5) PFGB_R(6) PFGB_R(7) PFGB_R(8) PFGB_R(9) PFGB_R(10) PFGB_R(11)
                PFGB_R(12) PFGB_R(13) PFGB_R(14) PFGB_R(15) PFGB_R(16)
#undef PFGB_R
            }
        }
        __syncthreads();
    }
}

template <>
__device__ void fft_lines_at<PFGB_LINE_T, PFGB_LINE_DIR>(LineTile t, const AxisPlan *plan) {
    run_stages<PFGB_LINE_T, PFGB_LINE_DIR>(t, *plan);
}
