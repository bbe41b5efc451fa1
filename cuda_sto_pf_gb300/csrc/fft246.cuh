// fft246.cuh — FP32 line transforms of length 246 = 6 x 41 for the grids
// whose axes are 246 long, and the three elastic-iteration passes built on
// them (y transform of six spectra, x transform + Green's operator, z
// C2R -> h_ij -> R2C).
//
// Cooley-Tukey with n = 41 n1 + n2 and k = k1 + 6 k2:
//   X[k1 + 6 k2] = sum_n2 W41^(n2 k2) W246^(n2 k1) sum_n1 x[41 n1 + n2] W6^(n1 k1)
// stage A: for each (line, n2) the 6-point DFT over n1, times W246^(n2 k1),
//          written back to the same six slots (position 41 k1 + n2);
// stage C: for each (line, k1) the 41-point DFT over n2 of positions
//          41 k1 .. 41 k1 + 40, written to positions k1 + 6 k2.
// Stage C is one 41-point DFT per thread by Rader's convolution in packed
// f32x2 arithmetic (dft41.cuh).  The stage is bound by instruction issue: the
// direct symmetric form's 1,600 multiply-adds took 78 us for 175,000 lines
// (two blocks per SM, the data in shared memory), the convolution's 350
// packed ones 48 us; in scalar instructions it took 59-62 us, and with the
// constants read from constant memory 80 us.
// A block holds NL lines and runs all NL * 6 stage-C items at once, one per
// thread: read, block barrier, write in place.
//
// What bounds a pass: a block loads its lines, transforms them and stores
// them, one after the other, so memory and arithmetic overlap only across the
// blocks of an SM.  The z passes, whose rows are contiguous, take four blocks
// of 21 lines per SM, the strided passes two of 42, whose row segments are
// longer.  Both are 16 warps in multiples of the register file's four-warp
// unit, which gives the 41-point stage 128 registers and no spills (48 lines
// in 9 warps left it 96: 78 instead of 58 us for the direct form, 48 instead
// of 40 us for the packed convolution, in the measurement above).
#pragma once

#include "dft41.cuh"
#include "fft.cuh"

namespace f246 {

constexpr int N = 246;
// blocks of the tensor-core forms (dft41_tc.cuh): three tiles of 128 items
constexpr int NL = 48;
constexpr int TC = NL / 6;        // columns per block of the strided-axis passes (even: 16-byte pairs)
constexpr int ZR = NL / 3;        // rows per block of the z pass
constexpr int THREADS = NL * 6;   // one stage-C item per thread
constexpr int BLOCKS_PER_SM = 96 / NL;

template <int NL_>
struct Eng {
    static constexpr int NL = NL_;
    static constexpr int ITEMS = NL * 6;
    static constexpr int THREADS = (ITEMS + 31) / 32 * 32;
    static constexpr int BLOCKS = NL <= 21 ? 4 : 2;
    // twiddles + the lines: positions x lines (strided axes) or lines x positions (z)
    static constexpr size_t SMEM = (size_t)(N + N * NL) * sizeof(float2);
    static_assert(THREADS * BLOCKS <= 512 || NL == 48, "registers");
    static_assert(SMEM * BLOCKS <= 220 * 1024, "blocks per SM");
};

// Lines-fast layout (LS = 1): element (line l, position p) at buf[p * PS + l]
// with PS = NL, so that the items of every stage walk consecutive addresses.
// Positions-fast layout (z): PS = 1, LS = N; stage C's items then have the odd
// stride 41.  Both are free of bank conflicts.

// stage A over NLT lines
template <int NLT, int DIR, int PS, int LS>
__device__ __forceinline__ void stage_a(float2 *buf, const float2 *tw) {
    constexpr int ITEMS = NLT * 41;
    for (int it = threadIdx.x; it < ITEMS; it += blockDim.x) {
        int l, n2;
        if (LS == 1) { n2 = it / NLT; l = it - n2 * NLT; }   // consecutive threads: consecutive lines
        else { l = it / 41; n2 = it - l * 41; }             // consecutive threads: consecutive positions
        float2 *b = buf + l * LS + n2 * PS;
        float2 v[6];
#pragma unroll
        for (int r = 0; r < 6; ++r) v[r] = b[41 * r * PS];
        bfly6<float, DIR>(v);
#pragma unroll
        for (int r = 1; r < 6; ++r) v[r] = twmul<DIR>(v[r], tw[n2 * r]);
#pragma unroll
        for (int r = 0; r < 6; ++r) b[41 * r * PS] = v[r];
    }
}

// stage C; contains the block barrier that separates its reads from its writes
template <int NLT, int DIR, int PS, int LS>
__device__ __forceinline__ void stage_c(float2 *buf) {
    const int it = threadIdx.x;
    const bool act = it < NLT * 6;
    int l, k1;
    if (LS == 1) { k1 = it / NLT; l = it - k1 * NLT; }
    else { l = it / 6; k1 = it - l * 6; }
    if (!act) { l = 0; k1 = 0; }
    float2 *b = buf + l * LS;
    d41::In v;
    d41::load(v, [&](int n) { return b[(41 * k1 + n) * PS]; });
    __syncthreads();
    if (!act) return;
    d41::store<DIR>(v, [&](int q, float2 x) { b[(k1 + 6 * q) * PS] = x; });
}

// full transform of the NLT lines in place; all threads of the block call it
template <int NLT, int DIR, int PS, int LS>
__device__ __forceinline__ void lines(float2 *buf, const float2 *tw) {
    stage_a<NLT, DIR, PS, LS>(buf, tw);
    __syncthreads();
    stage_c<NLT, DIR, PS, LS>(buf);
    __syncthreads();
}

__device__ __forceinline__ void load_twiddles(float2 *s, const float2 *g) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) s[i] = g[i];
}

// a tile of TCW columns x 246 positions between global memory (position
// stride es) and the lines-fast buffer (position stride PS): positions in
// [z0, z1) and columns past kcnt count as zero.  16-byte copies of column
// pairs where the tile is even, 8-byte ones where it is odd.
template <int TCW, int PS>
__device__ __forceinline__ void tile_in(float2 *buf, const float2 *src, long long es, int kcnt, int z0, int z1) {
    constexpr int V = TCW % 2 == 0 && PS % 2 == 0 ? 2 : 1;
    constexpr int TP = TCW / V;
    for (int e = threadIdx.x; e < N * TP; e += blockDim.x) {
        const int tp = e % TP, q = e / TP;
        const int t = V * tp;
        float2 *d = buf + q * PS + t;
        const float2 *s = src + (long long)q * es + t;
        const bool keep = q < z0 || q >= z1;
        if constexpr (V == 2) {
            if (keep && t + 1 < kcnt) {
                const unsigned sa = (unsigned)__cvta_generic_to_shared(d);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(s));
            } else {
                d[0] = keep && t < kcnt ? s[0] : make_float2(0.f, 0.f);
                d[1] = make_float2(0.f, 0.f);
            }
        } else {
            const bool ok = keep && t < kcnt;
            cp_async_elem(d, ok ? s : src, ok);
        }
    }
}
template <int TCW, int PS>
__device__ __forceinline__ void tile_out(const float2 *buf, float2 *dst, long long es, int kcnt, int z0, int z1) {
    constexpr int V = TCW % 2 == 0 && PS % 2 == 0 ? 2 : 1;
    constexpr int TP = TCW / V;
    for (int e = threadIdx.x; e < N * TP; e += blockDim.x) {
        const int tp = e % TP, q = e / TP;
        const int t = V * tp;
        if (q >= z0 && q < z1) continue;
        const float2 *s = buf + q * PS + t;
        float2 *d = dst + (long long)q * es + t;
        if (V == 2 && t + 1 < kcnt) *reinterpret_cast<float4 *>(d) = *reinterpret_cast<const float4 *>(s);
        else if (t < kcnt) d[0] = s[0];
    }
}

// z rows: NF half spectra of each of R rows (op.load_spec) packed as Hermitian
// pairs into the lines of a row, LW lines apart; only the kept columns are read
template <int NF, int LW, class Op>
__device__ __forceinline__ void rows_in(float2 *buf, const Op &op, long long row0, int R, int rcnt, int nk) {
    constexpr int LI = (NF + 1) / 2;
#pragma unroll 2
    for (int e = threadIdx.x; e < R * nk; e += blockDim.x) {
        const int rr = e / nk, k = e - rr * nk;
        float2 v[NF];
        if (rr < rcnt) op.load_spec(row0 + rr, k, v);
        else {
#pragma unroll
            for (int f = 0; f < NF; ++f) v[f] = make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int f = 0; f < LI; ++f) {
            float2 A = v[2 * f], B = 2 * f + 1 < NF ? v[2 * f + 1] : make_float2(0.f, 0.f);
            if (k == 0 || 2 * k == N) { A.y = 0.f; B.y = 0.f; }
            float2 *line = buf + (rr * LW + f) * N;
            // Z_k = A_k + i B_k ; Z_(n-k) = conj(A_k) + i conj(B_k)
            line[k] = make_float2(A.x - B.y, A.y + B.x);
            if (k > 0 && 2 * k != N) line[N - k] = make_float2(A.x + B.y, B.x - A.y);
        }
    }
    const int nz = N - 2 * nk + 1;   // positions nk .. N - nk hold no kept mode
    if (nz > 0)
        for (int e = threadIdx.x; e < R * LW * nz; e += blockDim.x) {
            const int l = e / nz;
            buf[l * N + nk + (e - l * nz)] = make_float2(0.f, 0.f);
        }
}
// the NF half spectra of each row from its packed lines to op.store_spec
template <int NF, int LW, class Op>
__device__ __forceinline__ void rows_out(const float2 *buf, const Op &op, long long row0, int rcnt, int nk) {
    constexpr int LO = (NF + 1) / 2;
    for (int e = threadIdx.x; e < rcnt * nk; e += blockDim.x) {
        const int rr = e / nk, k = e - rr * nk;
        float2 v[NF];
#pragma unroll
        for (int f = 0; f < LO; ++f) {
            const float2 *line = buf + (rr * LW + f) * N;
            const float2 Zk = line[k], Zm = line[k == 0 ? 0 : N - k];
            // A_k = (Z_k + conj Z_-k) / 2 ; B_k = (Z_k - conj Z_-k) / (2 i)
            v[2 * f] = make_float2(0.5f * (Zk.x + Zm.x), 0.5f * (Zk.y - Zm.y));
            if (2 * f + 1 < NF) v[2 * f + 1] = make_float2(0.5f * (Zk.y + Zm.y), 0.5f * (Zm.x - Zk.x));
        }
        op.store_spec(row0 + rr, k, v);
    }
}

constexpr int Y_NL = 42;          // columns per block of the elastic y pass

}  // namespace f246

// ---------------------------------------------------------------------------
// y-axis transform of six spectra in place.  Block (bx, i, s): spectrum s,
// columns kz = 42 bx .. 42 bx + 41 of x-plane i: 336-byte row segments, and
// two blocks cover the 82 kept columns of a 246-point z axis.  103 to 108 us per
// pass at 246^3; 121 us before the packed butterflies, when 21 columns in four
// blocks per SM took 127 us and three spectra of 16 columns in one block, 14 of
// every 96 lines empty, 133 us.
// ---------------------------------------------------------------------------
template <int DIR>
__global__ void __launch_bounds__(f246::Eng<f246::Y_NL>::THREADS, f246::Eng<f246::Y_NL>::BLOCKS)
k_y246(Grid3 g, const float2 *tw_g, AxisIO<float, 6, 6> io, const double *skip) {
    dependent_begin();
    if (skip && *skip != 0.0) return;
    using namespace f246;
    constexpr int NLT = Y_NL;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float2 *tw = reinterpret_cast<float2 *>(smem_raw);
    float2 *buf = tw + N;
    const int k0 = blockIdx.x * NLT, i = blockIdx.y;
    const int kcnt = min(NLT, g.NzK - k0);
    const long long base = (long long)i * N * g.NzC + k0;   // (i, y = 0, k0)
    // the array picked by selects, so that every io index is a compile-time
    // constant (a run-time index puts the struct in local memory)
    const float2 *in = io.in[0];
    float2 *out = io.out[0];
#pragma unroll
    for (int s = 1; s < 6; ++s)
        if ((int)blockIdx.z == s) { in = io.in[s]; out = io.out[s]; }
    tile_in<NLT, NLT>(buf, in + base, g.NzC, kcnt, DIR > 0 ? g.jc0 : N, DIR > 0 ? g.jc1 : N);
    cp_async_commit();
    load_twiddles(tw, tw_g);
    cp_async_wait_all();
    __syncthreads();
    lines<NLT, DIR, NLT, 1>(buf, tw);
    // the stage-C outputs are in natural order: position k of line l
    tile_out<NLT, NLT>(buf, out + base, g.NzC, kcnt, DIR < 0 ? g.jc0 : N, DIR < 0 ? g.jc1 : N);
}

// ---------------------------------------------------------------------------
// generic strided-axis pass on the 246-point engine: NIN spectra in, an
// optional forward transform (DIN), the op's per-point apply(i, j, k, in, out)
// in place, an optional inverse transform (DOUT), NOUT spectra out.  A block's
// lines are NW = max(NIN, NOUT) arrays x TCW columns.
// axis 1: y (block (bx, x-plane)); axis 2: x (block (bx, y-row)).  Lines
// beyond the NIN inputs are transformed too and never stored.
// ---------------------------------------------------------------------------
template <int NIN, int NOUT>
constexpr bool f246_axis_fits() {
    constexpr int NW = NIN > NOUT ? NIN : NOUT;
    return NW >= 1 && NW <= 6 && NW != 5;
}
// lines per block: 42 columns of one array, 21 of two, 14 of three, 10 of
// four, 7 of six
constexpr int f246_axis_lines(int NW) { return NW == 4 ? 40 : 42; }

template <int NIN, int NOUT, int DIN, int DOUT, class Op>
__global__ void __launch_bounds__(f246::Eng<f246_axis_lines(NIN > NOUT ? NIN : NOUT)>::THREADS,
                                  f246::Eng<f246_axis_lines(NIN > NOUT ? NIN : NOUT)>::BLOCKS)
k_axis246(Grid3 g, int axis, const float2 *tw_g, AxisIO<float, NIN, NOUT> io, Op op, const double *skip) {
    dependent_begin();
    if (skip && *skip != 0.0) return;
    using namespace f246;
    constexpr int NW = NIN > NOUT ? NIN : NOUT;
    constexpr int NLT = f246_axis_lines(NW), TCW = NLT / NW;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float2 *tw = reinterpret_cast<float2 *>(smem_raw);
    float2 *buf = tw + N;
    const int k0 = blockIdx.x * TCW, slab = axis == 1 ? blockIdx.y : g.kept_row(blockIdx.y);
    const int kcnt = min(TCW, g.NzK - k0);
    const int z0 = axis == 1 ? g.jc0 : N, z1 = axis == 1 ? g.jc1 : N;   // cut rows of a y pass
    long long base, es;
    if (axis == 1) { base = (long long)slab * N * g.NzC + k0; es = g.NzC; }
    else { base = (long long)slab * g.NzC + k0; es = (long long)g.Ny * g.NzC; }
#pragma unroll
    for (int s = 0; s < NIN; ++s) tile_in<TCW, NLT>(buf + s * TCW, io.in[s] + base, es, kcnt, DIN > 0 ? z0 : N, DIN > 0 ? z1 : N);
    cp_async_commit();
    if (DIN != 0 || DOUT != 0) load_twiddles(tw, tw_g);
    cp_async_wait_all();
    __syncthreads();
    if (DIN != 0) lines<NLT, DIN, NLT, 1>(buf, tw);
    if constexpr (!Op::kInplace) {
        if constexpr (op_has_begin<Op>::value) op.begin();
        for (int e = threadIdx.x; e < N * TCW; e += blockDim.x) {
            const int q = e / TCW, t = e % TCW;
            const int i = axis == 1 ? slab : q, j = axis == 1 ? q : slab;
            float2 vin[NIN > 0 ? NIN : 1], vout[NOUT > 0 ? NOUT : 1];
            float2 *pt = buf + q * NLT + t;
#pragma unroll
            for (int s = 0; s < NIN; ++s) vin[s] = pt[s * TCW];
            op.apply(i, j, min(k0 + t, g.NzC - 1), vin, vout);
#pragma unroll
            for (int s = 0; s < NOUT; ++s) pt[s * TCW] = vout[s];
        }
        __syncthreads();
    }
    if (DOUT != 0) lines<NLT, DOUT, NLT, 1>(buf, tw);
#pragma unroll
    for (int s = 0; s < NOUT; ++s) tile_out<TCW, NLT>(buf + s * TCW, io.out[s] + base, es, kcnt, DIN < 0 ? z0 : N, DIN < 0 ? z1 : N);
}
