// fft.cuh — shared-memory mixed-radix FFT engine and 3D pass kernels.
//
// The 3D real transform of a C-order [Nx][Ny][Nz] grid is done in three
// passes, each reading and writing the whole array once:
//   z pass : real rows (contiguous, length Nz) <-> half spectra (NzC = Nz/2+1)
//   y pass : complex lines of length Ny, element stride NzC
//   x pass : complex lines of length Nx, element stride Ny*NzC
// Each pass stages a tile of lines in shared memory and transforms them there
// in place (fft_lines below).  The passes take functors, so pointwise physics
// (RHS, flux, eigenstrain/h_ij, stress) runs inside the z pass, and the
// spectral updates (semi-implicit filters, gradients, Green's contraction) run
// inside the x pass between the forward and the inverse x transform.
//
// Real-data trick: two real lines a, b are transformed as one complex line
// z = a + i b;  A_k = (Z_k + conj Z_{N-k})/2, B_k = (Z_k - conj Z_{N-k})/(2i).
// The inverse packs two half spectra the same way; the imaginary parts of the
// k=0 and Nyquist bins are ignored (Hermitian input), like the C2R transform
// of the reference.
#pragma once

#include <algorithm>
#include <type_traits>
#include <utility>

#include "common.cuh"
#include "f32x2.cuh"
#include "rader41.cuh"

#define PFGB_MAX_STAGES 16
#define PFGB_MAX_N 1024
#define PFGB_LINE_THREADS 256   // threads of a generic pass's block at most
#define PFGB_DIRECT_SUMS 8      // sums of a direct stage that a thread holds

// Division by a run-time constant d via a multiply-high (round-up method):
// valid for every 32-bit dividend.
struct FastDiv {
    unsigned M;
    int L;
    unsigned d;
    __host__ __device__ void init(unsigned dd) {
        d = dd;
        if (d <= 1) { M = 0; L = 0; return; }
        L = 0;
        while ((1u << L) < d) ++L;
        M = (unsigned)((((unsigned long long)1 << 32) * ((1ull << L) - d)) / d + 1);
    }
    __device__ __forceinline__ unsigned div(unsigned x) const {
        if (d <= 1) return x;
        const unsigned t = __umulhi(M, x);
        return (t + ((x - t) >> 1)) >> (L - 1);
    }
};

// A thread's walk over rows of d elements, blockDim elements at a time: (q, l)
// advances by additions, with one division at the start.
struct Walk {
    int q, l, dq, dl, d;
    __device__ __forceinline__ explicit Walk(const FastDiv &f) {
        d = (int)f.d;
        q = (int)f.div(threadIdx.x);
        l = (int)threadIdx.x - q * d;
        dq = (int)f.div(blockDim.x);
        dl = (int)blockDim.x - dq * d;
    }
    __device__ __forceinline__ void step() {
        q += dq;
        l += dl;
        if (l >= d) { l -= d; ++q; }
    }
};

// One stage of a line transform of n points (decimation in frequency, in
// place): blocks of B points, B = R * m.  It takes the R points j' + r m of a
// block (j' < m), does their DFT, multiplies output r by W_B^(r j') and writes
// the outputs to the same R places.  The last stage (m = 1) writes them to
// their natural positions instead.
struct StagePlan {
    int R, B, m, kind;         // kind: 0 butterfly in registers, 1 Rader 41, 2 direct sums
    FastDiv fm, fR;
};

struct AxisPlan {
    int n;
    int nst;
    StagePlan st[PFGB_MAX_STAGES];
};

// radices of a line (1024 = 2^10: no length has more than ten factors); plans
// are made at C entries, which must not throw, so nothing here allocates
struct RadixList {
    int n = 0, r[10];
    void push(int f) { r[n++] = f; }
};

// host: the smooth part's radices in falling order, at most 16 each: as few
// stages as there can be, the largest radix as small as it can be
static inline void pfgb_best_radices(int q, int lim, RadixList &cur, RadixList &best) {
    if (q == 1) {
        if (!best.n || cur.n < best.n || (cur.n == best.n && cur.r[0] < best.r[0])) best = cur;
        return;
    }
    for (int r = std::min(lim, q); r >= 2; --r) {
        if (q % r) continue;
        cur.push(r);
        pfgb_best_radices(q / r, r, cur, best);
        --cur.n;
    }
}

// host: the stages of an n-point line, false if the kernels could not run
// them.  A factor 41 goes first (Rader's convolution), then the other primes
// above 13 as direct sums, then the smooth part with radices up to 16, the
// largest first.  The last butterfly stage holds a whole line, one butterfly
// per thread: where the smallest radix leaves it more than a block's threads
// (n / R > 256: 598 = 23 x 13 x 2), the largest smooth radix goes last, and
// where that is still too few points (n = 514, 578, 771, ...), a direct stage does,
// which holds eight sums per thread and so any n up to 2,048.
static inline bool pfgb_make_plan(int n, AxisPlan *p) {
    p->n = n;
    p->nst = 0;
    if (n < 1 || n > PFGB_MAX_N) return false;
    RadixList dir, cur, best;
    int q = n, B = n;
    auto stage = [&](int R, int kind) {
        StagePlan &st = p->st[p->nst++];
        st.R = R;
        st.kind = kind;
        st.B = B;
        st.m = B / R;
        st.fm.init((unsigned)st.m);
        st.fR.init((unsigned)R);
        B = st.m;
    };
    if (q % 41 == 0) { stage(41, 1); q /= 41; }
    for (int f = 17; f <= q; ++f)
        while (q % f == 0) {
            bool prime = true;
            for (int d = 2; d * d <= f; ++d) prime = prime && f % d;
            if (!prime) break;
            dir.push(f);
            q /= f;
        }
    if (q > 1) pfgb_best_radices(q, 16, cur, best);
    auto fits = [&] { return !best.n || n / best.r[best.n - 1] <= PFGB_LINE_THREADS; };
    if (!fits()) std::reverse(best.r, best.r + best.n);
    const bool direct_last = !fits();
    if (!direct_last) for (int i = 0; i < dir.n; ++i) stage(dir.r[i], 2);
    for (int i = 0; i < best.n; ++i) stage(best.r[i], 0);
    if (direct_last) for (int i = 0; i < dir.n; ++i) stage(dir.r[i], 2);
    for (int i = 0; i < p->nst; ++i) {
        const StagePlan &st = p->st[i];
        if (st.kind == 1 && i > 0) return false;
        if (st.kind == 2 && n > PFGB_LINE_THREADS * PFGB_DIRECT_SUMS) return false;
        if (st.kind == 0 && i == p->nst - 1 && n / st.R > PFGB_LINE_THREADS) return false;
    }
    return true;
}

// ---------------------------------------------------------------------------
// radix butterflies.  DIR = -1 forward (exp(-i..)), +1 inverse.
// ---------------------------------------------------------------------------
template <int DIR, typename T2> __device__ __forceinline__ T2 rot_mi(T2 a) {
    // forward: multiply by -i ; inverse: by +i
    return DIR < 0 ? mk2<T2>(a.y, -a.x) : mk2<T2>(-a.y, a.x);
}

// Sums within the butterflies; in FP32 one packed instruction for both parts,
// rounded as two.  Only for operands that are no products: the compiler cannot
// fuse a product into these, as it does into cadd and csub, and its own rounding
// would be one more.  pmad is k a + b, rounded once, for FP32's that are.  (With every
// sum packed the error of FP32 transforms with radices 3 to 9 was up to 7% larger.)
template <typename T2> __device__ __forceinline__ T2 padd(T2 a, T2 b) { return cadd(a, b); }
template <typename T2> __device__ __forceinline__ T2 psub(T2 a, T2 b) { return csub(a, b); }
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return f2x::un(f2x::add(f2x::pk(a), f2x::pk(b))); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return f2x::un(f2x::sub(f2x::pk(a), f2x::pk(b))); }
__device__ __forceinline__ float2 pmad(float2 a, float k, float2 b) {
    return f2x::un(f2x::fma(f2x::pk(a), f2x::both(k), f2x::pk(b)));
}

template <typename T, int DIR>
__device__ __forceinline__ void bfly2(cplx_t<T> *v) {
    auto a = v[0], b = v[1];
    v[0] = padd(a, b);
    v[1] = psub(a, b);
}
template <typename T, int DIR>
__device__ __forceinline__ void bfly4(cplx_t<T> *v) {
    auto t0 = padd(v[0], v[2]), t1 = psub(v[0], v[2]);
    auto t2 = padd(v[1], v[3]), t3 = rot_mi<DIR>(psub(v[1], v[3]));
    v[0] = padd(t0, t2);
    v[2] = psub(t0, t2);
    v[1] = padd(t1, t3);
    v[3] = psub(t1, t3);
}
template <typename T, int DIR>
__device__ __forceinline__ void bfly8(cplx_t<T> *v) {
    using T2 = cplx_t<T>;
    T2 e[4] = {v[0], v[2], v[4], v[6]};
    T2 o[4] = {v[1], v[3], v[5], v[7]};
    bfly4<T, DIR>(e);
    bfly4<T, DIR>(o);
    const T r = T(0.70710678118654752440084436210485);
    // W8^1 = r(1 -+ i), W8^2 = -+i, W8^3 = r(-1 -+ i)
    const T2 o2 = rot_mi<DIR>(o[2]), r1 = rot_mi<DIR>(o[1]), r3 = rot_mi<DIR>(o[3]);
    const T2 o1 = padd(o[1], r1), o3 = psub(r3, o[3]);
    v[0] = padd(e[0], o[0]); v[4] = psub(e[0], o[0]);
    v[2] = padd(e[2], o2);   v[6] = psub(e[2], o2);
    if constexpr (sizeof(T) == 4) {
        v[1] = pmad(o1, r, e[1]); v[5] = pmad(o1, -r, e[1]);
        v[3] = pmad(o3, r, e[3]); v[7] = pmad(o3, -r, e[3]);
    } else {
        v[1] = cadd(e[1], cscale(o1, r)); v[5] = csub(e[1], cscale(o1, r));
        v[3] = cadd(e[3], cscale(o3, r)); v[7] = csub(e[3], cscale(o3, r));
    }
}
template <typename T, int DIR>
__device__ __forceinline__ void bfly3(cplx_t<T> *v) {
    using T2 = cplx_t<T>;
    const T s3 = T(0.86602540378443864676372317075294);
    T2 a = v[0], s = padd(v[1], v[2]), d = psub(v[1], v[2]);
    const T2 m = mk2<T2>(a.x - T(0.5) * s.x, a.y - T(0.5) * s.y), r = rot_mi<DIR>(d);
    v[0] = padd(a, s);
    if constexpr (sizeof(T) == 4) {
        v[1] = pmad(r, s3, m);
        v[2] = pmad(r, -s3, m);
    } else {
        v[1] = cadd(m, cscale(r, s3));
        v[2] = csub(m, cscale(r, s3));
    }
}
template <typename T, int DIR>
__device__ __forceinline__ void bfly5(cplx_t<T> *v) {
    using T2 = cplx_t<T>;
    const T c1 = T(0.30901699437494742410229341718282);
    const T c2 = T(-0.80901699437494742410229341718282);
    const T s1 = T(0.95105651629515357211643933337938);
    const T s2 = T(0.58778525229247312916870595463907);
    T2 x0 = v[0];
    T2 a1 = padd(v[1], v[4]), b1 = psub(v[1], v[4]);
    T2 a2 = padd(v[2], v[3]), b2 = psub(v[2], v[3]);
    if constexpr (sizeof(T) == 4) {
        const T2 p1 = pmad(a2, c2, pmad(a1, c1, x0)), p2 = pmad(a2, c1, pmad(a1, c2, x0));
        const T2 r1 = rot_mi<DIR>(b1), r2 = rot_mi<DIR>(b2);
        v[0] = padd(padd(x0, a1), a2);
        v[1] = pmad(r1, s1, pmad(r2, s2, p1));
        v[4] = pmad(r1, -s1, pmad(r2, -s2, p1));
        v[2] = pmad(r1, s2, pmad(r2, -s1, p2));
        v[3] = pmad(r1, -s2, pmad(r2, s1, p2));
    } else {
        T2 p1 = mk2<T2>(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
        T2 p2 = mk2<T2>(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
        T2 q1 = rot_mi<DIR>(mk2<T2>(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y));
        T2 q2 = rot_mi<DIR>(mk2<T2>(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y));
        v[0] = mk2<T2>(x0.x + a1.x + a2.x, x0.y + a1.y + a2.y);
        v[1] = cadd(p1, q1);
        v[4] = csub(p1, q1);
        v[2] = cadd(p2, q2);
        v[3] = csub(p2, q2);
    }
}

// Asynchronous global->shared element copy (cp.async, sm_80+): all of a
// thread's tile loads are in flight at once.  `valid == false` zero-fills
// (source size 0; the source address is clamped to a valid one).
template <typename T2>
__device__ __forceinline__ void cp_async_elem(T2 *smem, const T2 *gmem, bool valid) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (sizeof(T2) == 16) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(valid ? 16 : 0));
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(valid ? 8 : 0));
    }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// twiddle w = W_n^e (table holds the forward roots); inverse uses conj
template <int DIR, typename T2>
__device__ __forceinline__ T2 twmul(T2 a, T2 w) {
    // the fused form written out, the same rounding wherever it is inlined
    const decltype(T2::x) wy = DIR < 0 ? w.y : -w.y;
    return mk2<T2>(fma(a.x, w.x, -(a.y * wy)), fma(a.y, w.x, a.x * wy));
}

template <typename T, int DIR>
__device__ __forceinline__ void bfly6(cplx_t<T> *v) {
    // 6 = 2 x 3: E = DFT3(x0,x2,x4), O = DFT3(x1,x3,x5), X_k = E_k + W6^k O_k
    using T2 = cplx_t<T>;
    T2 e[3] = {v[0], v[2], v[4]}, o[3] = {v[1], v[3], v[5]};
    bfly3<T, DIR>(e);
    bfly3<T, DIR>(o);
    // W6^1 = (1/2, -+ s3), W6^2 = (-1/2, -+ s3)
    const T h = T(0.5), s3 = T(0.86602540378443864676372317075294);
    v[0] = padd(e[0], o[0]); v[3] = psub(e[0], o[0]);
    if constexpr (sizeof(T) == 4) {
        const T2 r1 = rot_mi<DIR>(o[1]), r2 = rot_mi<DIR>(o[2]);
        v[1] = pmad(o[1], h, pmad(r1, s3, e[1]));    v[4] = pmad(o[1], -h, pmad(r1, -s3, e[1]));
        v[2] = pmad(o[2], -h, pmad(r2, s3, e[2]));   v[5] = pmad(o[2], h, pmad(r2, -s3, e[2]));
    } else {
        const T sg = DIR < 0 ? -s3 : s3;
        T2 o1 = mk2<T2>(h * o[1].x - sg * o[1].y, h * o[1].y + sg * o[1].x);
        T2 o2 = mk2<T2>(-h * o[2].x - sg * o[2].y, -h * o[2].y + sg * o[2].x);
        v[1] = cadd(e[1], o1);   v[4] = csub(e[1], o1);
        v[2] = cadd(e[2], o2);   v[5] = csub(e[2], o2);
    }
}

// ---------------------------------------------------------------------------
// Line transforms in shared memory, in place.  L lines of n points; element
// (line l, position p) at buf[p * PS + l * LS] (PS = L, LS = 1 for strided
// axes; PS = 1, LS odd for z rows).  The lanes of a warp walk the lines, so
// every access is contiguous in l (or has the odd stride LS): no bank
// conflicts at any stage but the last, whose chunks can be narrower than a
// warp, and the index arithmetic is per butterfly of up to 16 points.  A line
// makes one trip through shared memory per stage: at most two stages for most
// lengths up to 256 (125, 200, 243 and 13 others take three), at most three up
// to 1024 (625 and 875 take four).
//
// The transform is a device function of its own translation unit
// (fftline.cu), one per precision and direction: every pass kernel calls the
// same code, which is compiled once.  It takes shared-memory addresses, so
// that its accesses stay shared-memory instructions.
// ---------------------------------------------------------------------------
// the tile of a transform: shared addresses of the lines and of the twiddle
// table, the strides in bytes, the line count
struct LineTile {
    uint32_t buf, tw;
    int PS, LS;
    FastDiv fL;                // by the line count
};

template <typename T, int DIR> __device__ void fft_lines_at(LineTile t, const AxisPlan *plan);
template <> __device__ void fft_lines_at<float, -1>(LineTile, const AxisPlan *);
template <> __device__ void fft_lines_at<float, +1>(LineTile, const AxisPlan *);
template <> __device__ void fft_lines_at<double, -1>(LineTile, const AxisPlan *);
template <> __device__ void fft_lines_at<double, +1>(LineTile, const AxisPlan *);

// the whole transform of a tile's lines; all threads of the block call it,
// ends with __syncthreads()
template <typename T, int DIR>
__device__ __forceinline__ void fft_lines(const cplx_t<T> *buf, const cplx_t<T> *tw, const AxisPlan &p,
                                          const FastDiv &fL, int PS, int LS) {
    using T2 = cplx_t<T>;
    LineTile t;
    t.buf = (uint32_t)__cvta_generic_to_shared(buf);
    t.tw = (uint32_t)__cvta_generic_to_shared(tw);
    t.PS = PS * (int)sizeof(T2);
    t.LS = LS * (int)sizeof(T2);
    t.fL = fL;
    fft_lines_at<T, DIR>(t, &p);
}

// inputs of the direct sums that a point of a line goes through
static inline int pfgb_direct_inputs(const AxisPlan &p) {
    int d = 0;
    for (int s = 0; s < p.nst; ++s)
        if (p.st[s].kind == 2) d += p.st[s].R;
    return d;
}

// threads of a block whose tile has L lines: one trip of every stage where 256
// threads hold it, else equal trips (a second trip of a few butterflies would
// leave the block's other warps waiting).  The last stage has one butterfly per
// thread in registers, a direct stage eight sums, and both take whole lines.
static inline int pfgb_line_threads(const AxisPlan &p, int L) {
    int t = 64, least = 64;
    for (int s = 0; s < p.nst; ++s) {
        const int R = p.st[s].R, nb = p.n / R;
        int per = 1;                                   // work items of a thread and trip
        long long items = (long long)L * nb;
        if (p.st[s].kind == 1) items *= 8;             // eight lanes per butterfly
        else if (p.st[s].kind == 2) {
            items = (long long)L * p.n;
            per = PFGB_DIRECT_SUMS;
            least = std::max(least, (p.n + per - 1) / per);
            t = std::max(t, (int)std::min<long long>(items, PFGB_LINE_THREADS));   // fewer sums one after the other
        } else if (s == p.nst - 1) least = std::max(least, nb);
        const long long trips = (items + PFGB_LINE_THREADS * per - 1) / (PFGB_LINE_THREADS * per);
        t = std::max(t, (int)((items + trips * per - 1) / (trips * per)));
    }
    // (pfgb_make_plan keeps `least` within a block)
    return std::min(PFGB_LINE_THREADS, (std::max(t, least) + 31) / 32 * 32);
}

// blocks per SM that the pass kernels' registers allow for (80 or 128 per
// thread at 256 threads)
template <typename T> constexpr int pass_blocks() { return sizeof(T) == 4 ? 3 : 2; }

// load the twiddle table of length n into shared memory
template <typename T>
__device__ __forceinline__ void load_tw(cplx_t<T> *s, const cplx_t<T> *g, int n) {
#pragma unroll 1
    for (int i = threadIdx.x; i < n; i += blockDim.x) s[i] = g[i];
}

// 3D grid description passed to every pass kernel.  A solver's grid carries
// the 2/3 dealias rule as the box of modes it keeps: kz < NzK and ky rows
// outside [jc0, jc1).  Every x pass of the solver masks its result with that
// rule, so the passes around it move and transform only what the box holds:
// a z pass reads and writes the columns kz < NzK, a forward y pass writes and
// an inverse y pass reads the kept rows (the others count as zero), and an x
// pass runs over kept columns and rows alone.  What lies outside the box is
// never read.  That is 4/9 of an x pass and 2/3 of the columns elsewhere, with
// bitwise the results of the full passes.  Plain transforms keep everything
// (NzK = NzC, jc0 = jc1 = Ny).
struct Grid3 {
    int Nx, Ny, Nz, NzC;
    long long N, Nk;
    int NzK, jc0, jc1;
    __host__ void keep_all() { NzK = NzC; jc0 = jc1 = Ny; }
    __host__ __device__ int kept_rows() const { return Ny - (jc1 - jc0); }
    // spectral points of one array that a z pass (all rows) and an x pass
    // (kept rows) move
    __host__ double cols() const { return (double)Nx * Ny * NzK; }
    __host__ double kept() const { return (double)Nx * kept_rows() * NzK; }
    // the b-th kept ky row
    __device__ __forceinline__ int kept_row(int b) const { return b < jc0 ? b : b + (jc1 - jc0); }
    __device__ __forceinline__ bool cut_row(int j) const { return j >= jc0 && j < jc1; }
};

// ---------------------------------------------------------------------------
// Strided axis pass (y or x).  A block owns TK consecutive kz columns of one
// (i) slab (y pass) or one (j) slab (x pass): lines of length n, element
// stride `es`.  All NIN arrays of the tile sit interleaved in one shared
// buffer (row q holds max(NIN, NOUT) x TK values, array-major) and are
// transformed together with direction DIN (0 = none); op.apply(i, j, k, vin,
// vout) combines them point by point in place; the NOUT outputs are
// transformed together with DOUT (0 = none) and stored.  A pass with an
// identity op transforms each array by itself: one array per block
// (blockIdx.z), with as many more columns.
// ---------------------------------------------------------------------------
template <typename T, int NIN, int NOUT>
struct AxisIO {
    const cplx_t<T> *in[NIN > 0 ? NIN : 1];
    cplx_t<T> *out[NOUT > 0 ? NOUT : 1];
};

template <int NIN, int NOUT> constexpr int axis_width() { return NIN > NOUT ? NIN : NOUT; }

// ops may declare begin(): what a thread reads once before its points
template <class Op, class = void>
struct op_has_begin { static constexpr bool value = false; };
template <class Op>
struct op_has_begin<Op, std::void_t<decltype(std::declval<Op &>().begin())>> { static constexpr bool value = true; };

// divisors of an axis pass's loops: the columns of a tile, the lines that it
// transforms forward and back
struct TileDiv {
    FastDiv tk, in, out;
};

// arrays that share a block's tile
template <int NIN, int NOUT, class Op> constexpr int axis_tile_arrays() {
    return Op::kInplace ? 1 : axis_width<NIN, NOUT>();
}

template <typename T, int NIN, int NOUT, int DIN, int DOUT, class Op>
__global__ void __launch_bounds__(256, pass_blocks<T>())
k_axis_pass(Grid3 g, int axis, const __grid_constant__ AxisPlan plan, const cplx_t<T> *tw_g, TileDiv td,
            AxisIO<T, NIN, NOUT> io, Op op, const double *skip) {
    dependent_begin<T>();
    if (skip && *skip != 0.0) return;   // a finished elastic iteration: launched ahead, nothing to do
    using T2 = cplx_t<T>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T2 *sm = reinterpret_cast<T2 *>(smem_raw);
    constexpr bool INPL = Op::kInplace;   // identity op: outputs are the inputs
    constexpr int NW = axis_tile_arrays<NIN, NOUT, Op>();
    constexpr int NI = INPL ? 1 : NIN, NO = INPL ? 1 : NOUT;
    const FastDiv fTK = td.tk;
    const int n = plan.n, TK = (int)fTK.d, SP = NW * TK;
    T2 *tw = sm, *A = sm + n;

    const int k0 = blockIdx.x * TK;
    const int slab = axis == 1 ? blockIdx.y : g.kept_row(blockIdx.y);   // i for the y pass, j for the x pass
    long long base;
    int es;
    if (axis == 1) { base = (long long)slab * g.Ny * g.NzC + k0; es = g.NzC; }
    else { base = (long long)slab * g.NzC + k0; es = g.Ny * g.NzC; }
    const int kcnt = min(TK, g.NzK - k0);
    // rows cut by the dealias rule: zero into an inverse y pass, not written
    // by a forward one
    const int z0 = axis == 1 ? g.jc0 : n, z1 = axis == 1 ? g.jc1 : n;
    // the arrays of this block (selects: a run-time index of io would put it
    // in local memory)
    const T2 *in[NI > 0 ? NI : 1];
    T2 *out[NO > 0 ? NO : 1];
#pragma unroll
    for (int a = 0; a < NI; ++a) in[a] = io.in[a] + base;
#pragma unroll
    for (int a = 0; a < NO; ++a) out[a] = io.out[a] + base;
    if constexpr (INPL) {
#pragma unroll
        for (int a = 1; a < NIN; ++a)
            if ((int)blockIdx.z == a) { in[0] = io.in[a] + base; out[0] = io.out[a] + base; }
    }

    if (DIN != 0 || DOUT != 0) load_tw<T>(tw, tw_g, n);
    // (loops kept rolled here and below: a small grid runs each instruction
    // once or twice per block, and fetching unrolled code is what it waits for)
#pragma unroll 1
    for (Walk w(fTK); w.q < n; w.step()) {
        const bool ok = w.l < kcnt && !(DIN > 0 && w.q >= z0 && w.q < z1);
        const int o = ok ? w.q * es + w.l : 0;
#pragma unroll
        for (int a = 0; a < NI; ++a) cp_async_elem(&A[w.q * SP + a * TK + w.l], in[a] + o, ok);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (DIN != 0) fft_lines<T, DIN>(A, tw, plan, td.in, SP, 1);
    if constexpr (!INPL) {
        if constexpr (op_has_begin<Op>::value) op.begin();
#pragma unroll 1
        for (Walk w(fTK); w.q < n; w.step()) {
            const int q = w.q, l = w.l;
            const int k = min(k0 + l, g.NzC - 1);
            const int i = (axis == 1) ? slab : q;
            const int j = (axis == 1) ? q : slab;
            T2 vin[NI > 0 ? NI : 1], vout[NO > 0 ? NO : 1];
#pragma unroll
            for (int a = 0; a < NI; ++a) vin[a] = A[q * SP + a * TK + l];
            op.apply(i, j, k, vin, vout);
#pragma unroll
            for (int a = 0; a < NO; ++a) A[q * SP + a * TK + l] = vout[a];
        }
        __syncthreads();
    }
    if (DOUT != 0) fft_lines<T, DOUT>(A, tw, plan, td.out, SP, 1);
#pragma unroll 1
    for (Walk w(fTK); w.q < n; w.step()) {
        if (w.l < kcnt && !(DIN < 0 && w.q >= z0 && w.q < z1)) {
#pragma unroll
            for (int a = 0; a < NO; ++a) out[a][w.q * es + w.l] = A[w.q * SP + a * TK + w.l];
        }
    }
}

// ops of the z pass may declare kBatch > 1 with a Pre type, fetch(cell, pre)
// and point_with(cell, pre, in, out, acc): their global reads are then
// issued for kBatch cells of a thread at once
template <class Op, class = void>
struct op_batch { static constexpr int value = 1; };
template <class Op>
struct op_batch<Op, std::void_t<decltype(Op::kBatch)>> { static constexpr int value = Op::kBatch; };

// identity op for plain axis transforms
template <typename T, int NF>
struct OpCopy {
    static constexpr bool kInplace = true;
    __device__ __forceinline__ void apply(int, int, int, const cplx_t<T> *vin, cplx_t<T> *vout) const {
#pragma unroll
        for (int a = 0; a < NF; ++a) vout[a] = vin[a];
    }
};

// ---------------------------------------------------------------------------
// z pass: R consecutive rows per block.  Inputs: NFI half spectra per row
// (op.load_spec), inverse-transformed to real (C2R, unnormalised); then
// op.point(cell, in[NFI], out[NFO]) per cell; then NFO real fields are
// forward-transformed (R2C) and handed to op.store_spec(row, kz, v[NFO]).
// NFI = 0 makes it a pure R2C pass with a pointwise producer, NFO = 0 a pure
// C2R pass with a pointwise consumer.
// Real lines are paired (line 2p -> real part, 2p+1 -> imaginary part of
// complex line p); line index = row * NF + field.
// ---------------------------------------------------------------------------
// Reduction hook of the z pass: an op declares `struct Acc` with
// kActive, identity(), combine(a, b) and shuffle-able members (reduced with
// warp shuffles + shared memory, deterministic for a fixed launch shape).
struct NoAcc {
    static constexpr bool kActive = false;
    __device__ static NoAcc identity() { return NoAcc(); }
};

template <class Acc>
__device__ void block_reduce_acc(Acc &a) {
    __shared__ Acc red[32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a = Acc::combine(a, Acc::shfl_down(a, off));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = a;
    __syncthreads();
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        a = (lane < nw) ? red[lane] : Acc::identity();
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) a = Acc::combine(a, Acc::shfl_down(a, off));
    }
}

// divisors of the z pass's loops: Nz, NzC, the kept columns, the lines in and out
struct ZDiv {
    FastDiv n, nc, nk, in, out;
};

template <typename T, int NFI, int NFO, class Op>
__global__ void __launch_bounds__(256, 2)
k_zpass(Grid3 g, const __grid_constant__ AxisPlan plan, const cplx_t<T> *tw_g, int R, Op op, ZDiv zd,
        const double *skip) {
    dependent_begin<T>();
    if (skip && *skip != 0.0) return;
    using T2 = cplx_t<T>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T2 *sm = reinterpret_cast<T2 *>(smem_raw);
    const int n = g.Nz, nc = g.NzC, LS = n | 1;   // odd line stride: no bank conflicts across lines
    T2 *tw = sm;
    T2 *ws = sm + n;
    const int PI_ = (NFI > 0) ? (R * NFI + 1) / 2 : 0;
    const int PO_ = (NFO > 0) ? (R * NFO + 1) / 2 : 0;
    // NFI == NFO: the pointwise stage runs in place on the C2R result (same
    // line layout)
    constexpr bool SAME = (NFI == NFO);
    T2 *inA = ws, *outA = SAME ? ws : ws + PI_ * LS;
    const long long row0 = (long long)blockIdx.x * R;
    const long long nrows = (long long)g.Nx * g.Ny;
    const int rcnt = (int)min((long long)R, nrows - row0);
    load_tw<T>(tw, tw_g, n);

    auto pack = [&](int p, int k, T2 A, T2 B) {
        if (k == 0 || 2 * k == n) { A.y = T(0); B.y = T(0); }
        // Z_k = A_k + i B_k ; Z_{n-k} = conj(A_k) + i conj(B_k)
        inA[p * LS + k] = mk2<T2>(A.x - B.y, A.y + B.x);
        if (k > 0 && 2 * k != n) inA[p * LS + (n - k)] = mk2<T2>(A.x + B.y, B.x - A.y);
    };
    if (NFI > 0 && (NFI % 2) == 0) {
        // even field count: the pairs of a row are (f0,f1), (f2,f3), ...;
        // each (row, k) is loaded once
        for (Walk w(zd.nc); w.q < R; w.step()) {
            const int rr = w.q, k = w.l;
            T2 v[NFI > 0 ? NFI : 1];
            if (rr < rcnt && k < g.NzK) op.load_spec(row0 + rr, k, v);
            else {
#pragma unroll
                for (int f = 0; f < NFI; ++f) v[f] = mk2<T2>(T(0), T(0));
            }
#pragma unroll
            for (int f = 0; f < NFI / 2; ++f) pack(rr * (NFI / 2) + f, k, v[2 * f], v[2 * f + 1]);
        }
        __syncthreads();
        fft_lines<T, +1>(inA, tw, plan, zd.in, 1, LS);
    } else if (NFI > 0) {
        // pack pairs of half spectra into full complex spectra
        for (Walk w(zd.nc); w.q < PI_; w.step()) {
            const int p = w.q, k = w.l;
            T2 A = mk2<T2>(T(0), T(0)), B = mk2<T2>(T(0), T(0));
            const int la = 2 * p, lb = 2 * p + 1;
            const int ra = la / (NFI > 0 ? NFI : 1), fa = la - ra * (NFI > 0 ? NFI : 1);
            const int rb = lb / (NFI > 0 ? NFI : 1), fb = lb - rb * (NFI > 0 ? NFI : 1);
            T2 v[NFI > 0 ? NFI : 1];
            if (ra < rcnt && k < g.NzK) {
                op.load_spec(row0 + ra, k, v);
                A = v[fa];
                if (rb == ra) B = v[fb];
            }
            if (rb != ra && rb < rcnt && k < g.NzK) {
                op.load_spec(row0 + rb, k, v);
                B = v[fb];
            }
            pack(p, k, A, B);
        }
        __syncthreads();
        fft_lines<T, +1>(inA, tw, plan, zd.in, 1, LS);
    }
    // pointwise stage
    typename Op::Acc acc = Op::Acc::identity();
    auto cell_step = [&](int r, int z, auto &&pointf) {
        if (r >= rcnt) {
            if (NFO > 0) {
#pragma unroll
                for (int f = 0; f < NFO; ++f) {
                    const int l = r * NFO + f;
                    T *dst = reinterpret_cast<T *>(&outA[(l >> 1) * LS + z]);
                    dst[l & 1] = T(0);
                }
            }
            return;
        }
        T vi[NFI > 0 ? NFI : 1], vo[NFO > 0 ? NFO : 1];
#pragma unroll
        for (int f = 0; f < NFI; ++f) {
            const int l = r * NFI + f;
            const T *src = reinterpret_cast<const T *>(&inA[(l >> 1) * LS + z]);
            vi[f] = src[l & 1];
        }
        pointf((row0 + r) * n + z, vi, vo);
#pragma unroll
        for (int f = 0; f < NFO; ++f) {
            const int l = r * NFO + f;
            T *dst = reinterpret_cast<T *>(&outA[(l >> 1) * LS + z]);
            dst[l & 1] = vo[f];
        }
    };
    constexpr int B = op_batch<Op>::value;
    if constexpr (B > 1) {
        // the op's global reads of B cells go out together before any of
        // their stores (an op that reads and writes the same field cannot
        // have them reordered by the compiler)
        for (Walk w(zd.n); w.q < R;) {
            typename Op::Pre pre[B];
            int r[B], z[B];
#pragma unroll
            for (int b = 0; b < B; ++b) {
                r[b] = w.q;
                z[b] = w.l;
                if (w.q < rcnt) op.fetch((row0 + w.q) * n + w.l, pre[b]);
                w.step();
            }
#pragma unroll
            for (int b = 0; b < B; ++b)
                if (r[b] < R)
                    cell_step(r[b], z[b],
                              [&](long long cell, const T *vi, T *vo) { op.point_with(cell, pre[b], vi, vo, acc); });
        }
    } else {
        for (Walk w(zd.n); w.q < R; w.step())
            cell_step(w.q, w.l, [&](long long cell, const T *vi, T *vo) { op.point(cell, vi, vo, acc); });
    }
    if constexpr (Op::Acc::kActive) {
        block_reduce_acc(acc);
        if (threadIdx.x == 0) op.finish(blockIdx.x, acc);
    }
    if (NFO > 0) {
        // odd line count: zero the unused imaginary line
        if ((R * NFO) & 1) {
            const int l = R * NFO;
            for (int z = threadIdx.x; z < n; z += blockDim.x) {
                T *dst = reinterpret_cast<T *>(&outA[(l >> 1) * LS + z]);
                dst[1] = T(0);
            }
        }
        __syncthreads();
        fft_lines<T, -1>(outA, tw, plan, zd.out, 1, LS);
        // unpack and store: per (row, kz) gather all NFO fields
        for (Walk w(zd.nk); w.q < rcnt; w.step()) {
            const int rr = w.q, k = w.l;
            T2 v[NFO > 0 ? NFO : 1];
#pragma unroll
            for (int f = 0; f < NFO; ++f) {
                const int l = rr * NFO + f, p = l >> 1;
                const T2 Zk = outA[p * LS + k];
                const T2 Zm = outA[p * LS + (k == 0 ? 0 : n - k)];
                // A_k = (Z_k + conj Z_-k)/2 ; B_k = (Z_k - conj Z_-k)/(2i)
                if ((l & 1) == 0) v[f] = mk2<T2>(T(0.5) * (Zk.x + Zm.x), T(0.5) * (Zk.y - Zm.y));
                else v[f] = mk2<T2>(T(0.5) * (Zk.y + Zm.y), T(0.5) * (Zm.x - Zk.x));
            }
            op.store_spec(row0 + rr, k, v);
        }
    } else {
        __syncthreads();
    }
}
