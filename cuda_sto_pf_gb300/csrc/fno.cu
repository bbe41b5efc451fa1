// fno.cu — the learned warm start of the heterogeneous elastic iteration.
//
// A Fourier neural operator (FNO-3d of Li et al., ICLR 2021) maps
// (phi, eta, eps0 x 6) to the heterogeneous displacement correction
// u - u_hom.  The reference has no such model; it warm-starts from the
// previous step's displacement (main_cuda.cu:28792-28870).  The solver adds
// the prediction to the homogeneous solution and then runs the plain fixed
// point to its residual tolerance, so the model changes the starting point
// only, never the converged answer.
//
// Layout: activations are channel-major float [C][N], cell n = (x*Y + y)*Z + z.
// Weights (P, W_l, R_l, Q1, Q2) are read as bfloat16 from a copy of the
// float32 master vector; biases are read from the master vector.  All
// arithmetic is float32; weight-gradient sums over cells are float32 per
// block and combined across blocks in float64 in a fixed order, so results
// are run-to-run reproducible.
//
// The spectral convolution is a truncated DFT evaluated directly: with m
// retained modes per axis the transforms are dense (n x 2m) contractions,
// cheaper than full FFTs for m << n and exact on the retained set:
//   forward  z: real lines -> m half-spectrum coefficients (weight 1/N)
//            y, x: the two corner blocks [0,m) and [n-m,n)
//   mix      O[o][mode] = sum_i C[i][mode] R[i][o][mode]
//   inverse  x, y: expansion back to all n; z: c2r with weights 1, 2, 2, ...
// The backward pass uses the adjoints: each forward kernel's adjoint is the
// opposite-direction kernel with the weights exchanged.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "dfloat.cuh"
#include "f32x2.cuh"

namespace {

constexpr int kW = PFGB_FNO_WIDTH;     // 32
constexpr int kH = PFGB_FNO_HIDDEN;    // 64
constexpr int kIn = PFGB_FNO_IN;       // 8
constexpr int kOut = PFGB_FNO_OUT;     // 3
constexpr int kTile = 128;             // cells per tile of the backward kernels
constexpr int kRedBlocks = 4 * 152;    // blocks of the tiled backward kernels
constexpr int kMaxN = 1024;            // largest grid axis (as the solver)

#define FNO_TRY(x)                                                                       \
    do {                                                                                 \
        cudaError_t e_ = (x);                                                            \
        if (e_ != cudaSuccess) {                                                         \
            pfgb_set_error_msg("%s failed: %s (%s:%d)", #x, cudaGetErrorString(e_), __FILE__, \
                               __LINE__);                                                \
            return PFGB_ERR_CUDA;                                                        \
        }                                                                                \
    } while (0)
#define FNO_CHECK(x)                                   \
    do {                                               \
        pfgb_status s_ = (x);                          \
        if (s_ != PFGB_OK) return s_;                  \
    } while (0)

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}
__device__ __forceinline__ float bf(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float2 bf2(__nv_bfloat162 v) { return __bfloat1622float2(v); }

// corner-block index j in [0, 2m) -> wavenumber in [0, n)
__device__ __forceinline__ int kcorner(int j, int m, int n) { return j < m ? j : n - 2 * m + j; }

// ---------------------------------------------------------------------------
// lift: v0[o] = p[o] + sum_i P[o][i] * s_i a[i]
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_lift(const float *__restrict__ a, const __nv_bfloat16 *__restrict__ Pw,
                                              const float *__restrict__ pb, float4 s03, float4 s47,
                                              float *__restrict__ v0, long long N) {
    __shared__ float P[kW][kIn], b[kW];
    for (int e = threadIdx.x; e < kW * kIn; e += blockDim.x) P[e / kIn][e % kIn] = bf(Pw[e]);
    if (threadIdx.x < kW) b[threadIdx.x] = pb[threadIdx.x];
    __syncthreads();
    const float s[kIn] = {s03.x, s03.y, s03.z, s03.w, s47.x, s47.y, s47.z, s47.w};
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < N; n += (long long)gridDim.x * blockDim.x) {
        float x[kIn];
#pragma unroll
        for (int i = 0; i < kIn; ++i) x[i] = s[i] * a[i * N + n];
#pragma unroll 4
        for (int o = 0; o < kW; ++o) {
            float acc = b[o];
#pragma unroll
            for (int i = 0; i < kIn; ++i) acc = fmaf(P[o][i], x[i], acc);
            v0[o * N + n] = acc;
        }
    }
}

// ---------------------------------------------------------------------------
// z: dst[L][k] = w_k sum_z src[L][z] e^{-2 pi i k z / Z}, k < Mz
// (w_0 = w0, w_k = w1 for k > 0).  A thread sums 2 wavenumbers of 4 lines: per z
// one 16-byte read of the lines (staged transposed, kZC positions at a time)
// and one of the DFT matrix F[z][k] (k padded to even) feed 16 multiply-adds,
// eight packed ones.  Bound by issue: 128^3 x 32 lines, 12 modes, 300 us with
// one line per thread (two shared reads for four multiply-adds).
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int pad2(int m) { return (m + 1) & ~1; }
constexpr int kZC = 64;                // positions staged at a time
// lines per block: about 256 tasks (4 lines x 2 wavenumbers each)
__host__ __device__ constexpr int dft_z_lines(int Mz) {
    const int kg = pad2(Mz) / 2, g = 256 / kg;
    return 4 * (g > 42 ? 42 : (g < 1 ? 1 : g));
}
// row stride of the staged lines: an odd number of 16-byte words (conflict-free
// 16-byte stores by consecutive positions)
__host__ __device__ constexpr int dft_z_stride(int LB) { return (LB / 4) % 2 ? LB : LB + 4; }

__global__ void __launch_bounds__(256) k_dft_z(const float *__restrict__ src, float2 *__restrict__ dst,
                                               const float4 *__restrict__ fz, long long nlines, int Z, int Mz,
                                               int LB, float w0, float w1) {
    extern __shared__ __align__(16) float smz[];
    const int M2 = pad2(Mz), KG = M2 / 2, LS = dft_z_stride(LB), G4 = LB / 4;
    float4 *F4 = reinterpret_cast<float4 *>(smz);                // [kZC][KG]
    float *T = smz + 2 * kZC * M2;                               // [kZC][LS]
    const long long L0 = (long long)blockIdx.x * LB;
    const int nl = (int)min((long long)LB, nlines - L0);
    const float *s = src + L0 * Z;
    const int ntask = ((nl + 3) / 4) * KG;
    const int g = threadIdx.x / KG, q = threadIdx.x - g * KG;
    const bool act = (int)threadIdx.x < ntask;
    f2x::P acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = f2x::both(0.f);
    for (int zb = 0; zb < Z; zb += kZC) {
        const int nz = min(kZC, Z - zb);
        __syncthreads();
        for (int e = threadIdx.x; e < nz * KG; e += blockDim.x) F4[e] = fz[(long long)zb * KG + e];
        for (int e = threadIdx.x; e < kZC * G4; e += blockDim.x) {
            const int gg = e / kZC, z = e - gg * kZC;
            if (z < nz && 4 * gg < nl) {
                const float *p = s + (long long)(4 * gg) * Z + zb + z;
                float4 v;
                v.x = p[0];
                v.y = 4 * gg + 1 < nl ? p[Z] : 0.f;
                v.z = 4 * gg + 2 < nl ? p[2 * Z] : 0.f;
                v.w = 4 * gg + 3 < nl ? p[3 * Z] : 0.f;
                *reinterpret_cast<float4 *>(T + z * LS + 4 * gg) = v;
            }
        }
        __syncthreads();
        if (act) {
            const float *t = T + 4 * g;
#pragma unroll 4
            for (int z = 0; z < nz; ++z) {
                const float4 a = *reinterpret_cast<const float4 *>(t + z * LS);
                const float4 f = F4[z * KG + q];
                const f2x::P f0 = f2x::pk(make_float2(f.x, f.y)), f1 = f2x::pk(make_float2(f.z, f.w));
                const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const f2x::P b = f2x::both(av[i]);
                    acc[i][0] = f2x::fma(b, f0, acc[i][0]);
                    acc[i][1] = f2x::fma(b, f1, acc[i][1]);
                }
            }
        }
    }
    if (!act) return;
    const int k = 2 * q;
    const float wk = k == 0 ? w0 : w1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (4 * g + i >= nl) break;
        float2 *d = dst + (L0 + 4 * g + i) * Mz;
        const float2 c0 = f2x::un(acc[i][0]), c1 = f2x::un(acc[i][1]);
        d[k] = make_float2(c0.x * wk, c0.y * wk);
        if (k + 1 < Mz) d[k + 1] = make_float2(c1.x * w1, c1.y * w1);
    }
}

// y forward (e^{-}) onto the corner blocks: kYJ retained ky per thread share
// each value, NS slabs (channel, x) per block
// dst[r][jy][kz] = sum_y src[r][y][kz] e^{-2 pi i ky(jy) y / Y}
// tyi[jy][y] holds the conjugate twiddles; they are staged in shared memory,
// transposed, and read as broadcasts; the values come straight from memory.
// (Twiddles from the cache and slabs staged instead: the
// warps waited for the twiddles, 107 us at 128^3, 12 modes, issue 26%; now 48.)
constexpr int kYJ = 8, kYTab = 4096;
__host__ __device__ constexpr int dft_y_groups(int m) { return (2 * m + kYJ - 1) / kYJ; }
// positions whose twiddles fit
__host__ __device__ constexpr int dft_y_positions(int m) { return kYTab / (dft_y_groups(m) * kYJ); }
__global__ void __launch_bounds__(256) k_dft_y(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                               const float2 *__restrict__ tyi, long long nslab, int NS, int Y, int Mz,
                                               int m) {
    extern __shared__ __align__(16) float2 smy[];                // [Y][JP]
    const int J = 2 * m, JG = dft_y_groups(m), JP = JG * kYJ;
    const long long r0 = (long long)blockIdx.x * NS;
    const int ns = (int)min((long long)NS, nslab - r0), ntask = ns * Mz * JG;
    const float2 *s = src + r0 * Y * Mz;
    for (int i = threadIdx.x; i < Y * JP; i += blockDim.x) {
        const int j = i / Y, y = i - j * Y;
        smy[y * JP + j] = j < J ? tyi[j * Y + y] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    // kz fastest, then the slab: a warp shares the group of ky and its twiddles
    for (int e = threadIdx.x; e < ntask; e += blockDim.x) {
        const int jg = e / (ns * Mz), rem = e - jg * ns * Mz;
        const int sl = rem / Mz, kz = rem - sl * Mz;
        const float2 *a = s + (long long)sl * Y * Mz + kz;
        float re[kYJ], im[kYJ];
#pragma unroll
        for (int j = 0; j < kYJ; ++j) re[j] = im[j] = 0.f;
#pragma unroll 4
        for (int y = 0; y < Y; ++y) {
            const float2 v = a[y * Mz];
            const float4 *w = reinterpret_cast<const float4 *>(smy + y * JP + jg * kYJ);
#pragma unroll
            for (int q = 0; q < kYJ / 2; ++q) {                  // e^{-}: (tx, -ty)
                const float4 t = w[q];
                re[2 * q] = fmaf(v.x, t.x, fmaf(-v.y, -t.y, re[2 * q]));
                im[2 * q] = fmaf(v.x, -t.y, fmaf(v.y, t.x, im[2 * q]));
                re[2 * q + 1] = fmaf(v.x, t.z, fmaf(-v.y, -t.w, re[2 * q + 1]));
                im[2 * q + 1] = fmaf(v.x, -t.w, fmaf(v.y, t.z, im[2 * q + 1]));
            }
        }
        float2 *d = dst + (r0 + sl) * J * Mz + kz;
#pragma unroll
        for (int j = 0; j < kYJ; ++j)
            if (jg * kYJ + j < J) d[(jg * kYJ + j) * Mz] = make_float2(re[j], im[j]);
    }
}

// the same for few slabs: a block stages one, one output per thread
__global__ void __launch_bounds__(256) k_dft_y_slab(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                                    const float2 *__restrict__ twy, int Y, int Mz, int m) {
    extern __shared__ __align__(16) float2 smy[];
    float2 *tw = smy, *slab = smy + Y;
    const long long r = blockIdx.x;
    for (int e = threadIdx.x; e < Y; e += blockDim.x) tw[e] = twy[e];
    const float2 *s = src + r * Y * Mz;
    for (int e = threadIdx.x; e < Y * Mz; e += blockDim.x) slab[e] = s[e];
    __syncthreads();
    const int nout = 2 * m * Mz;
    for (int e = threadIdx.x; e < nout; e += blockDim.x) {
        const int jy = e / Mz, kz = e - jy * Mz;
        const int ky = kcorner(jy, m, Y);
        float re = 0.f, im = 0.f;
        int idx = 0;
        for (int y = 0; y < Y; ++y) {
            const float2 a = slab[y * Mz + kz], w = tw[idx];
            re = fmaf(a.x, w.x, fmaf(-a.y, w.y, re));
            im = fmaf(a.x, w.y, fmaf(a.y, w.x, im));
            idx += ky;
            if (idx >= Y) idx -= Y;
        }
        dst[r * nout + e] = make_float2(re, im);
    }
}

// x forward (e^{-}) onto the corner blocks: kXJ retained kx per thread share
// each value; block (channel, group of kx, chunk of q)
// dst[c][jx][q] = sum_x src[c][x][q] e^{-2 pi i kx(jx) x / X},  q < Q
// (One kx per block read the whole channel 2m times: 115 us at 128^3, 12 modes.)
constexpr int kXJ = 8, kXT = 96;
__global__ void __launch_bounds__(kXT) k_dft_x(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                               const float2 *__restrict__ twx, int X, int Q, int m) {
    extern __shared__ __align__(16) float2 smx[];                // [X][kXJ]
    const int J = 2 * m, c = blockIdx.y, j0 = blockIdx.z * kXJ, nj = min(kXJ, J - j0);
    for (int e = threadIdx.x; e < X * kXJ; e += blockDim.x) {
        const int x = e / kXJ, j = e - x * kXJ;
        smx[e] = j < nj ? twx[(int)(((long long)kcorner(j0 + j, m, X) * x) % X)] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int q = blockIdx.x * kXT + threadIdx.x;
    if (q >= Q) return;
    const float2 *s = src + (long long)c * X * Q + q;
    float re[kXJ], im[kXJ];
#pragma unroll
    for (int j = 0; j < kXJ; ++j) re[j] = im[j] = 0.f;
#pragma unroll 4
    for (int x = 0; x < X; ++x) {
        const float2 a = s[(long long)x * Q];
#pragma unroll
        for (int j = 0; j < kXJ; ++j) {
            const float2 w = smx[x * kXJ + j];
            re[j] = fmaf(a.x, w.x, fmaf(-a.y, w.y, re[j]));
            im[j] = fmaf(a.x, w.y, fmaf(a.y, w.x, im[j]));
        }
    }
#pragma unroll
    for (int j = 0; j < kXJ; ++j)
        if (j < nj) dst[((long long)c * J + j0 + j) * Q + q] = make_float2(re[j], im[j]);
}

// x inverse (e^{+}) from the corner blocks: one block per (channel, x)
// dst[c][x][q] = sum_jx src[c][jx][q] e^{+2 pi i kx(jx) x / X}
__global__ void __launch_bounds__(256) k_idft_x(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                                const float2 *__restrict__ twx, int X, int Q, int m) {
    __shared__ float2 w[128];   // 2m <= 128
    const int c = blockIdx.x / X, x = blockIdx.x % X;
    for (int j = threadIdx.x; j < 2 * m; j += blockDim.x) {
        const float2 t = twx[(int)(((long long)kcorner(j, m, X) * x) % X)];
        w[j] = make_float2(t.x, -t.y);
    }
    __syncthreads();
    const float2 *s = src + (long long)c * 2 * m * Q;
    for (int q = threadIdx.x; q < Q; q += blockDim.x) {
        float re = 0.f, im = 0.f;
#pragma unroll 8
        for (int j = 0; j < 2 * m; ++j) {
            const float2 a = s[(long long)j * Q + q], t = w[j];
            re = fmaf(a.x, t.x, fmaf(-a.y, t.y, re));
            im = fmaf(a.x, t.y, fmaf(a.y, t.x, im));
        }
        dst[((long long)c * X + x) * Q + q] = make_float2(re, im);
    }
}

// y inverse (e^{+}) from the corner blocks: eight positions per thread share
// each value, NS slabs (channel, x) and a chunk of positions per block
// dst[r][y][kz] = sum_jy src[r][jy][kz] e^{+2 pi i ky(jy) y / Y}
// tyi[jy][y] holds the twiddles (built once per model), staged in shared memory
// and read as broadcasts.  (One position per thread took a shared and a cached
// read for four multiply-adds: 72 us at 128^3, 12 modes; now 49.)
constexpr int kYP = 8;
__host__ __device__ constexpr int idft_y_chunk(int Y, int m) {
    const int c = kYTab / (2 * m) / kYP * kYP, p = (Y + kYP - 1) / kYP * kYP;
    return p < c ? p : c;
}
__global__ void __launch_bounds__(256) k_idft_y(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                                const float2 *__restrict__ tyi, long long nslab, int NS, int Y, int Mz,
                                                int m) {
    extern __shared__ __align__(16) float2 smiy[];               // [2m][YC]
    const int J = 2 * m, YC = idft_y_chunk(Y, m), yb = blockIdx.y * YC, ny = min(YC, Y - yb);
    const long long r0 = (long long)blockIdx.x * NS;
    const int ns = (int)min((long long)NS, nslab - r0), ntask = ns * Mz * ((ny + kYP - 1) / kYP);
    for (int i = threadIdx.x; i < J * YC; i += blockDim.x) {
        const int j = i / YC, y = i - j * YC;
        smiy[i] = y < ny ? tyi[j * Y + yb + y] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    // kz fastest, then the slab: a warp shares the positions and their twiddles
    for (int e = threadIdx.x; e < ntask; e += blockDim.x) {
        const int g = e / (ns * Mz), rem = e - g * ns * Mz;
        const int sl = rem / Mz, kz = rem - sl * Mz;
        const float2 *a = src + (r0 + sl) * J * Mz + kz;
        float re[kYP], im[kYP];
#pragma unroll
        for (int p = 0; p < kYP; ++p) re[p] = im[p] = 0.f;
#pragma unroll 4
        for (int j = 0; j < J; ++j) {
            const float2 v = a[j * Mz];
            const float4 *w = reinterpret_cast<const float4 *>(smiy + j * YC + g * kYP);
#pragma unroll
            for (int q = 0; q < kYP / 2; ++q) {
                const float4 t = w[q];
                re[2 * q] = fmaf(v.x, t.x, fmaf(-v.y, t.y, re[2 * q]));
                im[2 * q] = fmaf(v.x, t.y, fmaf(v.y, t.x, im[2 * q]));
                re[2 * q + 1] = fmaf(v.x, t.z, fmaf(-v.y, t.w, re[2 * q + 1]));
                im[2 * q + 1] = fmaf(v.x, t.w, fmaf(v.y, t.z, im[2 * q + 1]));
            }
        }
        float2 *d = dst + ((r0 + sl) * Y + yb + g * kYP) * Mz + kz;
#pragma unroll
        for (int p = 0; p < kYP; ++p)
            if (g * kYP + p < ny) d[p * Mz] = make_float2(re[p], im[p]);
    }
}

// the same for few slabs: a block stages one, one output per thread
__global__ void __launch_bounds__(256) k_idft_y_slab(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                                     const float2 *__restrict__ tyi, int Y, int Mz, int m) {
    extern __shared__ __align__(16) float2 smiy[];
    const long long r = blockIdx.x;
    const float2 *s = src + r * 2 * m * Mz;
    for (int e = threadIdx.x; e < 2 * m * Mz; e += blockDim.x) smiy[e] = s[e];
    __syncthreads();
    for (int e = threadIdx.x; e < Y * Mz; e += blockDim.x) {
        const int y = e / Mz, kz = e - y * Mz;
        float re = 0.f, im = 0.f;
#pragma unroll 4
        for (int j = 0; j < 2 * m; ++j) {
            const float2 a = smiy[j * Mz + kz];
            const float2 t = __ldg(&tyi[j * Y + y]);
            re = fmaf(a.x, t.x, fmaf(-a.y, t.y, re));
            im = fmaf(a.x, t.y, fmaf(a.y, t.x, im));
        }
        dst[r * (long long)Y * Mz + e] = make_float2(re, im);
    }
}

// O[o][md] = sum_i C[i][md] R[i][o][md]
__global__ void __launch_bounds__(256) k_mode_mix(const float2 *__restrict__ C, const __nv_bfloat162 *__restrict__ R,
                                                  float2 *__restrict__ O, int M) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)kW * M) return;
    const int o = (int)(e / M), md = (int)(e - (long long)o * M);
    float re = 0.f, im = 0.f;
#pragma unroll 8
    for (int i = 0; i < kW; ++i) {
        const float2 a = C[(long long)i * M + md];
        const float2 w = bf2(R[((long long)i * kW + o) * M + md]);
        re = fmaf(a.x, w.x, fmaf(-a.y, w.y, re));
        im = fmaf(a.x, w.y, fmaf(a.y, w.x, im));
    }
    O[e] = make_float2(re, im);
}

// adjoint of the mix: GC[i][md] = sum_o conj(R[i][o][md]) GO[o][md]
__global__ void __launch_bounds__(256) k_mode_mix_adj(const float2 *__restrict__ GO,
                                                      const __nv_bfloat162 *__restrict__ R, float2 *__restrict__ GC,
                                                      int M) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)kW * M) return;
    const int i = (int)(e / M), md = (int)(e - (long long)i * M);
    float re = 0.f, im = 0.f;
#pragma unroll 8
    for (int o = 0; o < kW; ++o) {
        const float2 g = GO[(long long)o * M + md];
        const float2 w = bf2(R[((long long)i * kW + o) * M + md]);
        re = fmaf(w.x, g.x, fmaf(w.y, g.y, re));
        im = fmaf(w.x, g.y, fmaf(-w.y, g.x, im));
    }
    GC[e] = make_float2(re, im);
}

// GR[i][o][md] (+)= conj(C[i][md]) GO[o][md]
__global__ void __launch_bounds__(256) k_mode_grad(const float2 *__restrict__ C, const float2 *__restrict__ GO,
                                                   float2 *__restrict__ GR, int M, int accumulate) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)kW * kW * M) return;
    const long long io = e / M;
    const int md = (int)(e - io * M);
    const int i = (int)(io / kW), o = (int)(io - (long long)i * kW);
    const float2 a = C[(long long)i * M + md], g = GO[(long long)o * M + md];
    float2 r = make_float2(a.x * g.x + a.y * g.y, a.x * g.y - a.y * g.x);
    if (accumulate) { const float2 p = GR[e]; r.x += p.x; r.y += p.y; }
    GR[e] = r;
}

// ---------------------------------------------------------------------------
// one spectral layer's output: z c2r of the mixed spectrum (weights 1, 2, 2,
// ...) fused with the pointwise path
//   pre[o] = spec[o] + b[o] + sum_i W[o][i] v[i];  vout = GELU(pre) or pre
// Two cells per thread (neighbours on one line when Z is even), 256 cells per
// block; the block stages the half-spectrum lines its cells lie on (at most
// 256/Z + 2 lines).  All 32 outputs of a cell are sums in registers, packed in
// pairs: 16 bytes of weights or of spectrum feed four or two pairs of
// multiply-adds for both cells.  (One cell per thread in scalar arithmetic was
// bound by its 640 broadcast reads per cell: 395 us at 128^3, 12 modes.)
// ---------------------------------------------------------------------------
constexpr int kLayerCells = 256;
__host__ __device__ constexpr int layer_lines(int Z) { return kLayerCells / Z + 2; }

enum { kCellsPair, kCellsApart, kCellsOne };
template <bool ACT, bool SAVE, int CELLS>
__global__ void __launch_bounds__(CELLS == kCellsOne ? kLayerCells : kLayerCells / 2, CELLS == kCellsOne ? 2 : 3) k_layer_fwd(const float2 *__restrict__ A,
                                                                  const float *__restrict__ v,
                                                                  const __nv_bfloat16 *__restrict__ Ww,
                                                                  const float *__restrict__ bw,
                                                                  float *__restrict__ vout, float *__restrict__ pre,
                                                                  const float2 *__restrict__ gz, long long S, int Z,
                                                                  int Mz) {
    extern __shared__ __align__(16) float sml[];
    float (*WT)[kW] = reinterpret_cast<float (*)[kW]>(sml);   // WT[i][o], rows read as float4 broadcasts
    float *bs = sml + kW * kW;
    float4 *At = reinterpret_cast<float4 *>(bs + kW);          // [line][k][pair of channels]: (re, re, im, im)
    const long long N = S * Z;
    const long long c0 = (long long)blockIdx.x * kLayerCells;
    const long long c1 = min(N, c0 + kLayerCells);
    const long long sf = c0 / Z;
    const int nl = (int)((c1 - 1) / Z - sf + 1);
    float2 *G = reinterpret_cast<float2 *>(At + layer_lines(Z) * Mz * (kW / 2));   // G[k][z] = c_k e(k z)
    for (int e = threadIdx.x; e < kW * kW; e += blockDim.x) WT[e % kW][e / kW] = bf(Ww[e]);
    if (threadIdx.x < kW) bs[threadIdx.x] = bw[threadIdx.x];
    for (int e = threadIdx.x; e < Mz * Z; e += blockDim.x) {
        const float2 t = gz[e];
        const float w = e < Z ? 1.f : 2.f;   // k = 0 once, the others with their conjugates
        G[e] = make_float2(w * t.x, w * t.y);
    }
    for (int e = threadIdx.x; e < kW * nl * Mz; e += blockDim.x) {
        const int c = e / (nl * Mz), rem = e - c * nl * Mz;
        const float2 a = A[(c * S + sf) * Mz + rem];
        float *d = reinterpret_cast<float *>(At + rem * (kW / 2) + (c >> 1)) + (c & 1);
        d[0] = a.x;
        d[2] = a.y;
    }
    __syncthreads();
    constexpr bool PAIR = CELLS == kCellsPair;
    const long long n0 = PAIR ? c0 + 2 * threadIdx.x : c0 + threadIdx.x, n1 = PAIR ? n0 + 1 : n0 + kLayerCells / 2;
    if (n0 >= c1) return;
    const bool two = CELLS != kCellsOne && n1 < c1;
    const int l0 = (int)(n0 / Z - sf), z0 = (int)(n0 % Z);
    const int l1 = PAIR || !two ? l0 : (int)(n1 / Z - sf), z1 = PAIR ? z0 + 1 : (two ? (int)(n1 % Z) : z0);
    f2x::P s0[kW / 2], s1[kW / 2];
#pragma unroll
    for (int p = 0; p < kW / 2; ++p) s0[p] = s1[p] = f2x::pk(make_float2(bs[2 * p], bs[2 * p + 1]));
#pragma unroll 8
    for (int i = 0; i < kW; ++i) {
        float x0, x1;
        if (PAIR) {
            const float2 t = *reinterpret_cast<const float2 *>(v + i * N + n0);
            x0 = t.x;
            x1 = t.y;
        } else {
            x0 = v[i * N + n0];
            x1 = two ? v[i * N + n1] : 0.f;
        }
        const f2x::P b0 = f2x::both(x0), b1 = f2x::both(x1);
        const float4 *w4 = reinterpret_cast<const float4 *>(WT[i]);
#pragma unroll
        for (int q = 0; q < kW / 4; ++q) {
            const float4 w = w4[q];
            const f2x::P wa = f2x::pk(make_float2(w.x, w.y)), wb = f2x::pk(make_float2(w.z, w.w));
            s0[2 * q] = f2x::fma(wa, b0, s0[2 * q]);
            s0[2 * q + 1] = f2x::fma(wb, b0, s0[2 * q + 1]);
            s1[2 * q] = f2x::fma(wa, b1, s1[2 * q]);
            s1[2 * q + 1] = f2x::fma(wb, b1, s1[2 * q + 1]);
        }
    }
    for (int k = 0; k < Mz; ++k) {
        const float2 t0 = G[k * Z + z0], t1 = G[k * Z + z1];
        const f2x::P x0 = f2x::both(t0.x), y0 = f2x::both(t0.y), x1 = f2x::both(t1.x), y1 = f2x::both(t1.y);
        const float4 *a0 = At + (l0 * Mz + k) * (kW / 2), *a1 = At + (l1 * Mz + k) * (kW / 2);
#pragma unroll
        for (int p = 0; p < kW / 2; ++p) {
            // Re(a e^{+i theta}) of two channels
            const float4 a = a0[p];
            s0[p] = f2x::fma(f2x::pk(make_float2(a.x, a.y)), x0,
                             f2x::fma(f2x::pk(make_float2(a.z, a.w)), y0, s0[p]));
            const float4 b = PAIR ? a : a1[p];
            s1[p] = f2x::fma(f2x::pk(make_float2(b.x, b.y)), x1,
                             f2x::fma(f2x::pk(make_float2(b.z, b.w)), y1, s1[p]));
        }
    }
#pragma unroll
    for (int o = 0; o < kW; ++o) {
        const float2 u0 = f2x::un(s0[o / 2]), u1 = f2x::un(s1[o / 2]);
        const float p0 = o & 1 ? u0.y : u0.x, p1 = o & 1 ? u1.y : u1.x;
        const float g0 = ACT ? gelu(p0) : p0, g1 = ACT ? gelu(p1) : p1;
        if (PAIR) {
            if (SAVE) *reinterpret_cast<float2 *>(pre + o * N + n0) = make_float2(p0, p1);
            *reinterpret_cast<float2 *>(vout + o * N + n0) = make_float2(g0, g1);
        } else {
            if (SAVE) pre[o * N + n0] = p0;
            vout[o * N + n0] = g0;
            if (two) {
                if (SAVE) pre[o * N + n1] = p1;
                vout[o * N + n1] = g1;
            }
        }
    }
}

// dst[c][n] += w_k-weighted z c2r of A (adjoint of the forward z transform);
// G[k][z] = w_k e(k z) in shared memory, consecutive z per warp
__global__ void __launch_bounds__(256) k_idft_z_acc(const float2 *__restrict__ A, float *__restrict__ dst,
                                                    const float2 *__restrict__ gz, long long S, int Z, int Mz,
                                                    int LB, float w0, float w1) {
    extern __shared__ __align__(16) float2 smc[];
    float2 *G = smc, *At = smc + Mz * Z;
    for (int e = threadIdx.x; e < Mz * Z; e += blockDim.x) {
        const float2 t = gz[e];
        const float wk = e < Z ? w0 : w1;
        G[e] = make_float2(wk * t.x, wk * t.y);
    }
    const long long s0 = (long long)blockIdx.x * LB;
    const int nl = (int)min((long long)LB, S - s0);
    for (int e = threadIdx.x; e < kW * nl * Mz; e += blockDim.x) {
        const int c = e / (nl * Mz), rem = e - c * nl * Mz;
        At[e] = A[(c * S + s0) * Mz + rem];
    }
    __syncthreads();
    const long long N = S * Z;
    for (int e = threadIdx.x; e < kW * nl * Z; e += blockDim.x) {
        const int c = e / (nl * Z), rem = e - c * nl * Z;
        const int l = rem / Z, z = rem - l * Z;
        const float2 *a = At + (c * nl + l) * Mz;
        float s = 0.f;
#pragma unroll 4
        for (int k = 0; k < Mz; ++k) {
            const float2 t = G[k * Z + z], v = a[k];
            s = fmaf(v.x, t.x, fmaf(v.y, t.y, s));
        }
        dst[c * N + (s0 + l) * Z + z] += s;
    }
}

// projection: y = out_scale (Q2 GELU(Q1 v + q1) + q2); two cells per thread,
// four pairs of hidden units of each at a time in packed arithmetic
__global__ void __launch_bounds__(128) k_project(const float *__restrict__ v, const __nv_bfloat16 *__restrict__ Q1w,
                                                 const float *__restrict__ q1, const __nv_bfloat16 *__restrict__ Q2w,
                                                 const float *__restrict__ q2, float4 os, float *__restrict__ y,
                                                 long long N) {
    __shared__ __align__(16) float Q1T[kW][kH];
    __shared__ float b1[kH], Q2[kOut][kH], b2[kOut];
    for (int e = threadIdx.x; e < kH * kW; e += blockDim.x) Q1T[e % kW][e / kW] = bf(Q1w[e]);
    for (int e = threadIdx.x; e < kOut * kH; e += blockDim.x) Q2[e / kH][e % kH] = bf(Q2w[e]);
    if (threadIdx.x < kH) b1[threadIdx.x] = q1[threadIdx.x];
    if (threadIdx.x < kOut) b2[threadIdx.x] = q2[threadIdx.x];
    __syncthreads();
    const long long half = (N + 1) / 2;   // cells n and n + half
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < half; n += (long long)gridDim.x * blockDim.x) {
        const bool two = n + half < N;
        const long long n1 = two ? n + half : n;
        float x[kW], z[kW];
#pragma unroll
        for (int i = 0; i < kW; ++i) { x[i] = v[i * N + n]; z[i] = v[i * N + n1]; }
        float o[kOut], p[kOut];
#pragma unroll
        for (int c = 0; c < kOut; ++c) o[c] = p[c] = b2[c];
#pragma unroll 1
        for (int j = 0; j < kH; j += 8) {
            f2x::P s[4], t[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) s[q] = t[q] = f2x::pk(make_float2(b1[j + 2 * q], b1[j + 2 * q + 1]));
#pragma unroll
            for (int i = 0; i < kW; ++i) {
                const float4 wa = *reinterpret_cast<const float4 *>(&Q1T[i][j]);
                const float4 wb = *reinterpret_cast<const float4 *>(&Q1T[i][j + 4]);
                const f2x::P w[4] = {f2x::pk(make_float2(wa.x, wa.y)), f2x::pk(make_float2(wa.z, wa.w)),
                                     f2x::pk(make_float2(wb.x, wb.y)), f2x::pk(make_float2(wb.z, wb.w))};
                const f2x::P bx = f2x::both(x[i]), bz = f2x::both(z[i]);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    s[q] = f2x::fma(w[q], bx, s[q]);
                    t[q] = f2x::fma(w[q], bz, t[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 a = f2x::un(s[q]), b = f2x::un(t[q]);
                const float ha = gelu(a.x), hb = gelu(a.y), ga = gelu(b.x), gb = gelu(b.y);
#pragma unroll
                for (int c = 0; c < kOut; ++c) {
                    o[c] = fmaf(Q2[c][j + 2 * q + 1], hb, fmaf(Q2[c][j + 2 * q], ha, o[c]));
                    p[c] = fmaf(Q2[c][j + 2 * q + 1], gb, fmaf(Q2[c][j + 2 * q], ga, p[c]));
                }
            }
        }
        y[n] = os.x * o[0];
        y[N + n] = os.y * o[1];
        y[2 * N + n] = os.z * o[2];
        if (two) {
            y[n1] = os.x * p[0];
            y[N + n1] = os.y * p[1];
            y[2 * N + n1] = os.z * p[2];
        }
    }
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
// sum of squares of the target, block partials in float64
__global__ void __launch_bounds__(256) k_sumsq(const float *__restrict__ t, long long n, double *__restrict__ part) {
    __shared__ double red[256];
    double s = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double x = t[i];
        s += x * x;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// fixed-order float64 sum of nb partials over a block of 256 threads
__device__ __forceinline__ double block_sum256(const double *__restrict__ part, int nb) {
    __shared__ double red[256];
    double s = 0.0;
    for (int b = threadIdx.x; b < nb; b += 256) s += part[b];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    return red[0];
}
__global__ void __launch_bounds__(256) k_sum_partials(const double *__restrict__ part, int nb, double *__restrict__ out) {
    const double s = block_sum256(part, nb);
    if (threadIdx.x == 0) out[0] = s;
}

// Projection backward with the loss L = sum (y - t)^2 / den.
// Per block partials (float): G_Q1 [64][32], g_q1 [64], G_Q2 [3][64], g_q2 [3]
// in that order (the flat layout of Q1 q1 Q2 q2); loss numerator in lpart.
// Bound by instruction issue (6,000 fused multiply-adds a cell, two
// blocks per SM).  A cell's 64 hidden values stay in its row of the tile and the
// 32 outputs of g_v in registers, so that the loops over hidden units stay
// rolled (with the hidden values in registers they were 100 KB of code, 236
// registers; 64^3: 343 -> 241 us), and the bias and Q2 sums run along with the weights' loop.
constexpr int kProjE = kH * kW + kH + kOut * kH + kOut;   // 2307
constexpr int kVS = kW + 4;                               // v tile row stride (16-byte rows)
__host__ __device__ constexpr size_t project_bwd_smem_floats() {
    return (size_t)kH * kW + kOut * kH + kH + 4 + (size_t)kTile * (2 * (kH + 1) + kVS + 4);
}
__global__ void __launch_bounds__(kTile) k_project_bwd(const float *__restrict__ v, const float *__restrict__ tgt,
                                                       const __nv_bfloat16 *__restrict__ Q1w,
                                                       const float *__restrict__ q1,
                                                       const __nv_bfloat16 *__restrict__ Q2w,
                                                       const float *__restrict__ q2, float4 os,
                                                       const double *__restrict__ den, float *__restrict__ gv,
                                                       float *__restrict__ part, double *__restrict__ lpart,
                                                       long long N, long long ntiles) {
    extern __shared__ __align__(16) float smp[];
    float (*Q1)[kW] = reinterpret_cast<float (*)[kW]>(smp);                   // [64][32]
    float (*Q2)[kH] = reinterpret_cast<float (*)[kH]>(smp + kH * kW);
    float *b1 = smp + kH * kW + kOut * kH;
    float *b2 = b1 + kH;
    float (*Vs)[kVS] = reinterpret_cast<float (*)[kVS]>(b2 + 4);             // v tile (16-byte rows)
    float (*Gs)[kH + 1] = reinterpret_cast<float (*)[kH + 1]>(&Vs[kTile][0]); // hpre, then g_hpre tile
    float (*Hs)[kH + 1] = reinterpret_cast<float (*)[kH + 1]>(&Gs[kTile][0]); // h tile
    float (*Ys)[4] = reinterpret_cast<float (*)[4]>(&Hs[kTile][0]);           // g_y tile
    __shared__ double lred[kTile];
    const int t = threadIdx.x;
    for (int e = t; e < kH * kW; e += blockDim.x) Q1[e / kW][e % kW] = bf(Q1w[e]);
    for (int e = t; e < kOut * kH; e += blockDim.x) Q2[e / kH][e % kH] = bf(Q2w[e]);
    if (t < kH) b1[t] = q1[t];
    if (t < kOut) b2[t] = q2[t];
    __syncthreads();
    const float inv = (float)(1.0 / den[0]);
    const float osc[kOut] = {os.x, os.y, os.z};
    // owned entries: G_Q1[j][i0 .. i0+16), G_Q2 entries t and t + 128 (< 192)
    const int jo = t >> 1, i0 = (t & 1) * 16;
    float a1[16], a2[2] = {0.f, 0.f}, ab1 = 0.f, ab2 = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) a1[k] = 0.f;
    double lsum = 0.0;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long n = tile * kTile + t;
        const bool ok = n < N;
        float x[kW];
#pragma unroll
        for (int i = 0; i < kW; ++i) x[i] = ok ? v[i * N + n] : 0.f;
        float y[kOut];
#pragma unroll
        for (int c = 0; c < kOut; ++c) y[c] = b2[c];
#pragma unroll 2
        for (int j = 0; j < kH; ++j) {
            float s = b1[j];
            const float4 *w4 = reinterpret_cast<const float4 *>(Q1[j]);
#pragma unroll
            for (int q = 0; q < kW / 4; ++q) {
                const float4 w = w4[q];
                s = fmaf(w.x, x[4 * q], s);
                s = fmaf(w.y, x[4 * q + 1], s);
                s = fmaf(w.z, x[4 * q + 2], s);
                s = fmaf(w.w, x[4 * q + 3], s);
            }
            Gs[t][j] = s;   // hpre for now
            const float h = gelu(s);
            Hs[t][j] = ok ? h : 0.f;
#pragma unroll
            for (int c = 0; c < kOut; ++c) y[c] = fmaf(Q2[c][j], h, y[c]);
        }
        float gy[kOut];
#pragma unroll
        for (int c = 0; c < kOut; ++c) {
            const float r = ok ? osc[c] * y[c] - tgt[c * N + n] : 0.f;
            lsum += (double)r * (double)r;
            gy[c] = 2.f * r * inv * osc[c];
            Ys[t][c] = gy[c];
        }
        float sg[kW];
#pragma unroll
        for (int i = 0; i < kW; ++i) sg[i] = 0.f;
#pragma unroll 2
        for (int j = 0; j < kH; ++j) {
            float gh = 0.f;
#pragma unroll
            for (int c = 0; c < kOut; ++c) gh = fmaf(Q2[c][j], gy[c], gh);
            const float gj = ok ? gh * gelu_d(Gs[t][j]) : 0.f;
            Gs[t][j] = gj;
            const float4 *w4 = reinterpret_cast<const float4 *>(Q1[j]);
#pragma unroll
            for (int q = 0; q < kW / 4; ++q) {
                const float4 w = w4[q];
                sg[4 * q] = fmaf(w.x, gj, sg[4 * q]);
                sg[4 * q + 1] = fmaf(w.y, gj, sg[4 * q + 1]);
                sg[4 * q + 2] = fmaf(w.z, gj, sg[4 * q + 2]);
                sg[4 * q + 3] = fmaf(w.w, gj, sg[4 * q + 3]);
            }
        }
        if (ok) {
#pragma unroll
            for (int i = 0; i < kW; ++i) gv[i * N + n] = sg[i];
        }
#pragma unroll
        for (int i = 0; i < kW; ++i) Vs[t][i] = x[i];
        __syncthreads();
        float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
        for (int c = 0; c < kTile; ++c) {
            const float gj = Gs[c][jo];
            const float4 *v4 = reinterpret_cast<const float4 *>(&Vs[c][i0]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 w = v4[q];
                a1[4 * q] = fmaf(gj, w.x, a1[4 * q]);
                a1[4 * q + 1] = fmaf(gj, w.y, a1[4 * q + 1]);
                a1[4 * q + 2] = fmaf(gj, w.z, a1[4 * q + 2]);
                a1[4 * q + 3] = fmaf(gj, w.w, a1[4 * q + 3]);
            }
            ab1 += gj;
            s0 = fmaf(Ys[c][t / kH], Hs[c][t % kH], s0);
            if (t < kH) s1 = fmaf(Ys[c][2], Hs[c][t], s1);
            else if (t < kH + kOut) ab2 += Ys[c][t - kH];
        }
        a2[0] += s0;
        a2[1] += s1;
        __syncthreads();
    }
    float *P = part + (long long)blockIdx.x * kProjE;
#pragma unroll
    for (int k = 0; k < 16; ++k) P[jo * kW + i0 + k] = a1[k];
    if (t % 2 == 0) P[kH * kW + jo] = ab1;
    for (int r = 0; r < 2; ++r) {
        const int e = t + r * kTile;
        if (e < kOut * kH) P[kH * kW + kH + e] = a2[r];
    }
    if (t >= kH && t < kH + kOut) P[kH * kW + kH + kOut * kH + t - kH] = ab2;
    lred[t] = lsum;
    __syncthreads();
    if (t == 0) {
        double s = 0.0;
        for (int i = 0; i < kTile; ++i) s += lred[i];
        lpart[blockIdx.x] = s;
    }
}

// Pointwise backward of one layer: g_pre = g_out * act'(pre); g_v = W^T g_pre
// (the spectral adjoint is added later); per block partials of G_W [32][32]
// and g_b [32] (the flat layout of W_l b_l).  Eight channels at a time: their
// reads go out together and their part of g_v is added at once, so that the
// channels' loop stays rolled (unrolled, with erf in every channel, it was 40 KB
// of code; 64^3: 171 -> 74 us).
constexpr int kLayerE = kW * kW + kW;   // 1056
template <bool LAST>
__global__ void __launch_bounds__(kTile) k_layer_bwd(const float *__restrict__ gout, const float *__restrict__ pre,
                                                     const float *__restrict__ v, const __nv_bfloat16 *__restrict__ Ww,
                                                     float *__restrict__ gpre, float *__restrict__ gv,
                                                     float *__restrict__ part, long long N, long long ntiles) {
    __shared__ __align__(16) float Wm[kW][kW];
    __shared__ float Gs[kTile][kW + 1];
    __shared__ __align__(16) float Vs[kTile][kVS];
    const int t = threadIdx.x;
    for (int e = t; e < kW * kW; e += blockDim.x) Wm[e / kW][e % kW] = bf(Ww[e]);
    __syncthreads();
    const int oo = t >> 2, i0 = (t & 3) * 8;
    float aw[8], ab = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) aw[k] = 0.f;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long n = tile * kTile + t;
        const bool ok = n < N;
        float sg[kW];
#pragma unroll
        for (int i = 0; i < kW; ++i) sg[i] = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < kW; c0 += 8) {
            float x[8], p[8], y[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                x[u] = ok ? gout[(c0 + u) * N + n] : 0.f;
                p[u] = ok && !LAST ? pre[(c0 + u) * N + n] : 0.f;
                y[u] = ok ? v[(c0 + u) * N + n] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (!LAST) x[u] *= gelu_d(p[u]);
                if (ok) gpre[(c0 + u) * N + n] = x[u];
                Gs[t][c0 + u] = x[u];
                Vs[t][c0 + u] = y[u];
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float4 *w4 = reinterpret_cast<const float4 *>(Wm[c0 + u]);
#pragma unroll
                for (int q = 0; q < kW / 4; ++q) {
                    const float4 w = w4[q];
                    sg[4 * q] = fmaf(w.x, x[u], sg[4 * q]);
                    sg[4 * q + 1] = fmaf(w.y, x[u], sg[4 * q + 1]);
                    sg[4 * q + 2] = fmaf(w.z, x[u], sg[4 * q + 2]);
                    sg[4 * q + 3] = fmaf(w.w, x[u], sg[4 * q + 3]);
                }
            }
        }
        if (ok) {
#pragma unroll
            for (int i = 0; i < kW; ++i) gv[i * N + n] = sg[i];
        }
        __syncthreads();
#pragma unroll 4
        for (int c = 0; c < kTile; ++c) {
            const float go = Gs[c][oo];
            const float4 va = *reinterpret_cast<const float4 *>(&Vs[c][i0]);
            const float4 vb = *reinterpret_cast<const float4 *>(&Vs[c][i0 + 4]);
            aw[0] = fmaf(go, va.x, aw[0]); aw[1] = fmaf(go, va.y, aw[1]);
            aw[2] = fmaf(go, va.z, aw[2]); aw[3] = fmaf(go, va.w, aw[3]);
            aw[4] = fmaf(go, vb.x, aw[4]); aw[5] = fmaf(go, vb.y, aw[5]);
            aw[6] = fmaf(go, vb.z, aw[6]); aw[7] = fmaf(go, vb.w, aw[7]);
            ab += go;
        }
        __syncthreads();
    }
    float *P = part + (long long)blockIdx.x * kLayerE;
#pragma unroll
    for (int k = 0; k < 8; ++k) P[oo * kW + i0 + k] = aw[k];
    if (t % 4 == 0) P[kW * kW + oo] = ab;
}

// lift backward: G_P [32][8] and g_p [32] (the flat layout of P p)
constexpr int kLiftE = kW * kIn + kW;   // 288
__global__ void __launch_bounds__(kTile) k_lift_bwd(const float *__restrict__ g0, const float *__restrict__ a,
                                                    float4 s03, float4 s47, float *__restrict__ part, long long N,
                                                    long long ntiles) {
    __shared__ float Gs[kTile][kW + 1], As[kTile][kIn + 1];
    const int t = threadIdx.x;
    const float s[kIn] = {s03.x, s03.y, s03.z, s03.w, s47.x, s47.y, s47.z, s47.w};
    const int oo = t >> 2, i0 = (t & 3) * 2;
    float aw[2] = {0.f, 0.f}, ab = 0.f;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long n = tile * kTile + t;
        const bool ok = n < N;
#pragma unroll
        for (int c = 0; c < kW; ++c) Gs[t][c] = ok ? g0[c * N + n] : 0.f;
#pragma unroll
        for (int i = 0; i < kIn; ++i) As[t][i] = ok ? s[i] * a[i * N + n] : 0.f;
        __syncthreads();
        for (int c = 0; c < kTile; ++c) {
            const float go = Gs[c][oo];
            aw[0] = fmaf(go, As[c][i0], aw[0]);
            aw[1] = fmaf(go, As[c][i0 + 1], aw[1]);
        }
        if (t < kW) for (int c = 0; c < kTile; ++c) ab += Gs[c][t];
        __syncthreads();
    }
    float *P = part + (long long)blockIdx.x * kLiftE;
    P[oo * kIn + i0] = aw[0];
    P[oo * kIn + i0 + 1] = aw[1];
    if (t < kW) P[kW * kIn + t] = ab;
}

// grad[e] (+)= sum over blocks of part[b][e], float64, fixed order: a warp's
// lanes take 32 entries, the block's 32 warps every 32nd partial (608 partials
// of 2,307 entries: 98 us with one thread per entry, a chain of 608 loads)
__global__ void __launch_bounds__(1024) k_reduce_part(const float *__restrict__ part, int nb, int E,
                                                      float *__restrict__ grad, int accumulate) {
    __shared__ double red[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (e < E)
        for (int b = w; b < nb; b += 32) s += (double)part[(long long)b * E + e];
    red[w][lane] = s;
    __syncthreads();
    if (w == 0 && e < E) {
        double t = red[0][lane];
        for (int k = 1; k < 32; ++k) t += red[k][lane];
        grad[e] = accumulate ? (float)((double)grad[e] + t) : (float)t;
    }
}

// loss = sum(lpart) / den
__global__ void __launch_bounds__(256) k_loss_final(const double *__restrict__ lpart, int nb,
                                                    const double *__restrict__ den, double *__restrict__ out) {
    const double s = block_sum256(lpart, nb);
    if (threadIdx.x == 0) out[0] = s / den[0];
}

__global__ void __launch_bounds__(256) k_sumsq_f(const float *__restrict__ g, long long n, double *__restrict__ part) {
    __shared__ double red[256];
    // a thread's sum on the FP32 pipe, to more bits than a double's and over its
    // range (in FP64, whose pipe is 64 times slower, a conversion and a multiply-add
    // per entry take 70 us for 17M entries)
    fsum s = fs_zero();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        fs_add_square(s, g[i]);
    red[threadIdx.x] = fs_to_double(s);
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// Adam with decoupled weight decay on the float32 master weights; the
// bfloat16 copy is refreshed.  gscale = min(1, clip / ||g||) when clip > 0, once
// a block (its FP64 square root and quotient in every thread took 30 us).  Bound
// by memory, 30 bytes a weight: four weights a thread and trip.
__global__ void __launch_bounds__(256) k_adam(float *__restrict__ w, __nv_bfloat16 *__restrict__ wb,
                                              const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                                              long long n, float lr, float b1, float b2, float eps, float wd,
                                              float bc1, float bc2, float clip, const double *__restrict__ gnorm2) {
    __shared__ float gsh;
    if (threadIdx.x == 0) {
        gsh = 1.f;
        if (clip > 0.f) {
            const double nrm = sqrt(gnorm2[0]);
            if (nrm > (double)clip) gsh = (float)((double)clip / nrm);
        }
    }
    __syncthreads();
    const float gs = gsh;
    auto one = [&](float &wi, float g0, float &mi, float &vi) {
        const float gi = g0 * gs;
        mi = b1 * mi + (1.f - b1) * gi;
        vi = b2 * vi + (1.f - b2) * gi * gi;
        const float mh = mi / bc1, vh = vi / bc2;
        wi = wi - lr * (mh / (sqrtf(vh) + eps) + wd * wi);
    };
    const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
    for (long long q = i0; q < n / 4; q += st) {
        float4 w4 = reinterpret_cast<const float4 *>(w)[q], m4 = reinterpret_cast<const float4 *>(m)[q],
               v4 = reinterpret_cast<const float4 *>(v)[q];
        const float4 g4 = reinterpret_cast<const float4 *>(g)[q];
        one(w4.x, g4.x, m4.x, v4.x);
        one(w4.y, g4.y, m4.y, v4.y);
        one(w4.z, g4.z, m4.z, v4.z);
        one(w4.w, g4.w, m4.w, v4.w);
        reinterpret_cast<float4 *>(m)[q] = m4;
        reinterpret_cast<float4 *>(v)[q] = v4;
        reinterpret_cast<float4 *>(w)[q] = w4;
        reinterpret_cast<__nv_bfloat162 *>(wb)[2 * q] = __floats2bfloat162_rn(w4.x, w4.y);
        reinterpret_cast<__nv_bfloat162 *>(wb)[2 * q + 1] = __floats2bfloat162_rn(w4.z, w4.w);
    }
    for (long long i = n / 4 * 4 + i0; i < n; i += st) {
        one(w[i], g[i], m[i], v[i]);
        wb[i] = __float2bfloat16_rn(w[i]);
    }
}

__global__ void __launch_bounds__(256) k_to_bf16(const float *__restrict__ w, __nv_bfloat16 *__restrict__ wb, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        wb[i] = __float2bfloat16_rn(w[i]);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
uint64_t splitmix(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
double uniform01(uint64_t &s) { return (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0); }

}  // namespace

struct pfgb_fno {
    pfgb_fno_config cfg;
    int device = 0;
    cudaStream_t stream = nullptr;
    int X = 0, Y = 0, Z = 0, m = 0, L = 0, Mz = 0, Q = 0;
    long long N = 0, S = 0, M = 0, nparams = 0;
    long long offP = 0, offp = 0, offQ1 = 0, offq1 = 0, offQ2 = 0, offq2 = 0;
    std::vector<long long> offW, offb, offR;
    float *master = nullptr;
    __nv_bfloat16 *wbf = nullptr;
    float2 *twx = nullptr, *twy = nullptr;
    float2 *tyi = nullptr;   // [2m][Y] inverse y twiddles of the retained ky
    float4 *fz = nullptr;    // [Z][pad2(m)] e^{-2 pi i k z / Z}, read as float4 pairs of k
    float2 *gz = nullptr;    // [m][Z] the same values, z fastest
    // inference
    float *va = nullptr, *vb = nullptr;
    float2 *A = nullptr, *B = nullptr, *C = nullptr, *O = nullptr;
    // training
    bool train = false;
    std::vector<float *> vs, pres;
    std::vector<float2 *> Cs;
    float *G[3] = {nullptr, nullptr, nullptr};
    float *grad = nullptr, *am = nullptr, *av = nullptr, *part = nullptr;
    double *dpart = nullptr, *dscal = nullptr;
    long long adam_t = 0;
    std::vector<void *> allocs;
};

namespace {

pfgb_status fno_alloc(pfgb_fno *f, void **p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        pfgb_set_error_msg("FNO: cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
        return PFGB_ERR_CUDA;
    }
    f->allocs.push_back(*p);
    return PFGB_OK;
}
template <typename T>
pfgb_status fno_alloc_t(pfgb_fno *f, T **p, size_t count) {
    return fno_alloc(f, reinterpret_cast<void **>(p), sizeof(T) * count);
}

pfgb_status upload_tw(pfgb_fno *f, float2 **dst, int n) {
    std::vector<float2> h(n);
    for (int j = 0; j < n; ++j) {
        const double a = -2.0 * PFGB_PI * (double)j / (double)n;
        h[j] = make_float2((float)cos(a), (float)sin(a));
    }
    FNO_CHECK(fno_alloc_t(f, dst, n));
    FNO_TRY(cudaMemcpy(*dst, h.data(), sizeof(float2) * n, cudaMemcpyHostToDevice));
    return PFGB_OK;
}

constexpr size_t kSmemCap = 200 * 1024;
size_t layer_smem(int Z, int Mz);
// The models that are taken: those whose y pass can stage a slab (k_dft_y_slab),
// whose layer kernel its lines, and whose z pass could stage the DFT matrix of a
// whole line with about 256 / (modes / 2) lines (64 KB at most), within kSmemCap.
// The z pass stages less than that (kZC positions: at most 64 KB); the set of
// accepted models stayed.
size_t dft_z_staging(int Z, int Mz) {
    const int kg = pad2(Mz) / 2;
    const int lb = std::max(1, std::min((256 + kg - 1) / kg, (64 * 1024) / (4 * (Z + 1))));
    return sizeof(float) * (2 * (size_t)Z * pad2(Mz) + (size_t)lb * (Z + 1));
}
size_t layer_staging(int Z, int Mz) {
    return sizeof(float) * ((size_t)kW * kW + kW) +
           sizeof(float2) * ((size_t)Mz * Z + (size_t)kW * layer_lines(Z) * Mz);
}

pfgb_status validate(const pfgb_fno_config *c) {
    const int m = c->modes;
    if (c->Nx < 2 || c->Ny < 2 || c->Nz < 2 || c->Nx > kMaxN || c->Ny > kMaxN || c->Nz > kMaxN) {
        pfgb_set_error_msg("FNO: grid %dx%dx%d outside [2..%d]", c->Nx, c->Ny, c->Nz, kMaxN);
        return PFGB_ERR_INVALID;
    }
    if (m < 1 || m > 64 || 2 * m > c->Nx || 2 * m > c->Ny || 2 * m > c->Nz) {
        pfgb_set_error_msg("FNO: modes=%d needs 1 <= modes <= 64 and 2*modes <= Nx, Ny, Nz (%d, %d, %d)", m, c->Nx,
                           c->Ny, c->Nz);
        return PFGB_ERR_INVALID;
    }
    if (dft_z_staging(c->Nz, m) > kSmemCap || sizeof(float2) * (size_t)c->Ny * (m + 1) > kSmemCap) {
        pfgb_set_error_msg("FNO: modes=%d too many for a %dx%dx%d grid (shared-memory staging)", m, c->Nx, c->Ny,
                           c->Nz);
        return PFGB_ERR_UNSUPPORTED;
    }
    if (layer_staging(c->Nz, m) > kSmemCap) {
        pfgb_set_error_msg("FNO: modes=%d too many for Nz=%d (shared-memory staging)", m, c->Nz);
        return PFGB_ERR_UNSUPPORTED;
    }
    if (c->layers < 1 || c->layers > 16) {
        pfgb_set_error_msg("FNO: layers=%d outside [1, 16]", c->layers);
        return PFGB_ERR_INVALID;
    }
    for (int i = 0; i < kIn; ++i)
        if (!std::isfinite(c->in_scale[i])) { pfgb_set_error_msg("FNO: non-finite in_scale"); return PFGB_ERR_INVALID; }
    for (int i = 0; i < kOut; ++i)
        if (!std::isfinite(c->out_scale[i])) { pfgb_set_error_msg("FNO: non-finite out_scale"); return PFGB_ERR_INVALID; }
    return PFGB_OK;
}

void layout_offsets(pfgb_fno *f) {
    long long o = 0;
    f->offP = o; o += kW * kIn;
    f->offp = o; o += kW;
    f->offW.resize(f->L); f->offb.resize(f->L); f->offR.resize(f->L);
    for (int l = 0; l < f->L; ++l) {
        f->offW[l] = o; o += kW * kW;
        f->offb[l] = o; o += kW;
        f->offR[l] = o; o += (long long)kW * kW * f->M * 2;
    }
    f->offQ1 = o; o += kH * kW;
    f->offq1 = o; o += kH;
    f->offQ2 = o; o += kOut * kH;
    f->offq2 = o; o += kOut;
    f->nparams = o;
}

// seeded initial weights: U(-1/sqrt(fan_in), 1/sqrt(fan_in)) for the dense
// maps and biases; the spectral weights scale * U(0, 1) with scale = 1/W^2
void init_params(pfgb_fno *f, std::vector<float> &h) {
    h.assign((size_t)f->nparams, 0.f);
    uint64_t s = f->cfg.seed;
    auto fill = [&](long long off, long long n, double lo, double hi) {
        for (long long i = 0; i < n; ++i) h[(size_t)(off + i)] = (float)(lo + (hi - lo) * uniform01(s));
    };
    const double bi = 1.0 / sqrt((double)kIn), bw = 1.0 / sqrt((double)kW), bh = 1.0 / sqrt((double)kH);
    fill(f->offP, kW * kIn, -bi, bi);
    fill(f->offp, kW, -bi, bi);
    for (int l = 0; l < f->L; ++l) {
        fill(f->offW[l], kW * kW, -bw, bw);
        fill(f->offb[l], kW, -bw, bw);
        fill(f->offR[l], (long long)kW * kW * f->M * 2, 0.0, 1.0 / (kW * kW));
    }
    fill(f->offQ1, kH * kW, -bw, bw);
    fill(f->offq1, kH, -bw, bw);
    fill(f->offQ2, kOut * kH, -bh, bh);
    fill(f->offq2, kOut, -bh, bh);
}

int lines_per_block(int Z) { return std::max(1, 256 / Z); }

pfgb_status check_launch(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        pfgb_set_error_msg("FNO: %s launch failed: %s", what, cudaGetErrorString(e));
        return PFGB_ERR_CUDA;
    }
    return PFGB_OK;
}

template <typename K>
pfgb_status smem_opt_in(K kern, size_t bytes) {
    if (bytes <= 48 * 1024) return PFGB_OK;
    // one fixed value, the same from every caller: the limit belongs to the kernel,
    // and another model's smaller one could come between this and the launch
    FNO_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap));
    return PFGB_OK;
}

size_t dft_z_smem(int Mz, int LB) {
    return sizeof(float) * (2 * (size_t)kZC * pad2(Mz) + (size_t)kZC * dft_z_stride(LB));
}

// The forms for few threads.  k_dft_y and k_idft_y give a thread eight sums, whose
// chain of reads from memory needs 15 warps an SM beside it to be hidden, and
// k_dft_y the twiddles of all positions at once; k_layer_fwd gives a thread two cells,
// which below a block an SM only leaves threads out.  Either side gives the same
// results.  us a pass, eight sums / one (two cells / one), 4 layers:
//   y forward  12 modes: 56^3 -> 2.1 more, 64^3 1.1 less, 128^3 16 less; 8 modes: 64^3
//              6.6, 128^3 13 more; 4 modes: 8x1000x16 172 more; 24 modes (Y > chunk): 96^3 7.6 more
//   y inverse   8 modes: 32^3 4.2 more, 48^3 1.4, 64^3 4.3 less; 4 modes: 64^3 1.9 more
//   layer      24^3 to 32^3 1 to 2.6 more, 40^3 0.4 to 2, 64^3 6 less
constexpr long long kFewThreads = 152 * 480, kFewCells = 152 * kLayerCells;
bool few_slabs_fwd(const pfgb_fno *f) {
    return (long long)kW * f->X * f->Mz * dft_y_groups(f->m) < kFewThreads || f->Y > dft_y_positions(f->m);
}
bool few_slabs_inv(const pfgb_fno *f) {
    return (long long)kW * f->X * f->Mz * ((f->Y + kYP - 1) / kYP) < kFewThreads;
}
bool few_cells(const pfgb_fno *f) { return f->N <= kFewCells; }

// spectral transform of src [W][N] onto the retained modes -> dst [W][M]
pfgb_status spec_forward(pfgb_fno *f, const float *src, float2 *dst, float w0, float w1) {
    const long long lines = (long long)kW * f->S;
    // fewer lines per block where the grid would leave SMs without two blocks
    // (4 modes, 16x8x1000: 138 -> 79 us; 32x32x512 23 us less)
    const int LB = std::min(dft_z_lines(f->Mz), (int)std::max<long long>(4, lines / 304 / 4 * 4));
    const size_t sz = dft_z_smem(f->Mz, LB);
    FNO_CHECK(smem_opt_in(k_dft_z, sz));
    k_dft_z<<<(unsigned)((lines + LB - 1) / LB), 256, sz, f->stream>>>(src, f->A, f->fz, lines, f->Z, f->Mz, LB,
                                                                       w0, w1);
    FNO_CHECK(check_launch("dft_z"));
    if (few_slabs_fwd(f)) {
        const size_t sy = sizeof(float2) * ((size_t)f->Y + (size_t)f->Y * f->Mz);
        FNO_CHECK(smem_opt_in(k_dft_y_slab, sy));
        k_dft_y_slab<<<(unsigned)(kW * f->X), 256, sy, f->stream>>>(f->A, f->B, f->twy, f->Y, f->Mz, f->m);
    } else {
        // slabs per block: about 256 tasks, fewer where the grid would leave SMs
        // without two blocks
        const int tasks = f->Mz * dft_y_groups(f->m);
        const long long nslab = (long long)kW * f->X;
        const int NS = (int)std::max<long long>(1, std::min<long long>(256 / std::max(1, tasks), nslab / 304));
        const int ny_thr = std::min(256, (NS * tasks + 31) / 32 * 32);
        const size_t sy = sizeof(float2) * (size_t)f->Y * dft_y_groups(f->m) * kYJ;
        k_dft_y<<<(unsigned)((nslab + NS - 1) / NS), ny_thr, sy, f->stream>>>(f->A, f->B, f->tyi, nslab, NS, f->Y, f->Mz,
                                                                             f->m);
    }
    FNO_CHECK(check_launch("dft_y"));
    const size_t sx = sizeof(float2) * (size_t)f->X * kXJ;
    FNO_CHECK(smem_opt_in(k_dft_x, sx));
    k_dft_x<<<dim3((f->Q + kXT - 1) / kXT, kW, (2 * f->m + kXJ - 1) / kXJ), kXT, sx, f->stream>>>(f->B, dst, f->twx,
                                                                                              f->X, f->Q, f->m);
    return check_launch("dft_x");
}

// expansion of src [W][M] back to all x and y: -> f->A [W][S][Mz]
pfgb_status spec_inverse_xy(pfgb_fno *f, const float2 *src) {
    k_idft_x<<<(unsigned)(kW * f->X), 256, 0, f->stream>>>(src, f->B, f->twx, f->X, f->Q, f->m);
    FNO_CHECK(check_launch("idft_x"));
    if (few_slabs_inv(f)) {
        const size_t sy = sizeof(float2) * (2 * (size_t)f->m * f->Mz);
        FNO_CHECK(smem_opt_in(k_idft_y_slab, sy));
        k_idft_y_slab<<<(unsigned)(kW * f->X), 256, sy, f->stream>>>(f->B, f->A, f->tyi, f->Y, f->Mz, f->m);
        return check_launch("idft_y");
    }
    // slabs per block: a few trips over the staged twiddles, fewer where the grid
    // would leave SMs without four blocks
    const int YC = idft_y_chunk(f->Y, f->m), tasks = f->Mz * (YC / kYP);
    const long long nslab = (long long)kW * f->X;
    const int NS = (int)std::max<long long>(1, std::min<long long>(768 / tasks, nslab / 608));
    k_idft_y<<<dim3((unsigned)((nslab + NS - 1) / NS), (f->Y + YC - 1) / YC), std::min(256, (NS * tasks + 31) / 32 * 32),
               sizeof(float2) * 2 * (size_t)f->m * YC, f->stream>>>(f->B, f->A, f->tyi, nslab, NS, f->Y, f->Mz, f->m);
    return check_launch("idft_y");
}

size_t layer_smem(int Z, int Mz) { return layer_staging(Z, Mz); }

unsigned grid_cells(long long N) { return (unsigned)std::min<long long>((N + 255) / 256, 152LL * 16); }

pfgb_status forward_impl(pfgb_fno *f, const float *in, float *out, bool train) {
    const float *is = f->cfg.in_scale, *osc = f->cfg.out_scale;
    const float4 s03 = make_float4(is[0], is[1], is[2], is[3]), s47 = make_float4(is[4], is[5], is[6], is[7]);
    float *v = train ? f->vs[0] : f->va;
    k_lift<<<grid_cells(f->N), 256, 0, f->stream>>>(in, f->wbf + f->offP, f->master + f->offp, s03, s47, v, f->N);
    FNO_CHECK(check_launch("lift"));
    const float invN = (float)(1.0 / (double)f->N);
    const size_t sl = layer_smem(f->Z, f->Mz);
    for (int l = 0; l < f->L; ++l) {
        float *vin = train ? f->vs[l] : (l % 2 == 0 ? f->va : f->vb);
        float *vout = train ? f->vs[l + 1] : (l % 2 == 0 ? f->vb : f->va);
        float2 *C = train ? f->Cs[l] : f->C;
        FNO_CHECK(spec_forward(f, vin, C, invN, invN));
        const long long nm = (long long)kW * f->M;
        k_mode_mix<<<(unsigned)((nm + 255) / 256), 256, 0, f->stream>>>(
            C, reinterpret_cast<const __nv_bfloat162 *>(f->wbf + f->offR[l]), f->O, (int)f->M);
        FNO_CHECK(check_launch("mode_mix"));
        FNO_CHECK(spec_inverse_xy(f, f->O));
        const bool act = l < f->L - 1;
        const unsigned nb = (unsigned)((f->N + kLayerCells - 1) / kLayerCells);
        const bool one = few_cells(f);
        const int threads = one ? kLayerCells : kLayerCells / 2;
        auto launch = [&](auto kern) -> pfgb_status {
            FNO_CHECK(smem_opt_in(kern, sl));
            kern<<<nb, threads, sl, f->stream>>>(f->A, vin, f->wbf + f->offW[l], f->master + f->offb[l], vout,
                                                 train ? f->pres[l] : nullptr, f->gz, f->S, f->Z, f->Mz);
            return check_launch("layer_fwd");
        };
        auto cells = [&](auto form) -> pfgb_status {
            constexpr int C = decltype(form)::value;
            if (act) return train ? launch(k_layer_fwd<true, true, C>) : launch(k_layer_fwd<true, false, C>);
            return train ? launch(k_layer_fwd<false, true, C>) : launch(k_layer_fwd<false, false, C>);
        };
        if (one) FNO_CHECK(cells(std::integral_constant<int, kCellsOne>{}));
        else if (f->Z % 2 == 0) FNO_CHECK(cells(std::integral_constant<int, kCellsPair>{}));
        else FNO_CHECK(cells(std::integral_constant<int, kCellsApart>{}));
    }
    if (!out) return PFGB_OK;   // training: the projection backward recomputes it
    const float *vl = train ? f->vs[f->L] : (f->L % 2 == 0 ? f->va : f->vb);
    k_project<<<grid_cells(f->N), 128, 0, f->stream>>>(vl, f->wbf + f->offQ1, f->master + f->offq1,
                                                       f->wbf + f->offQ2, f->master + f->offq2,
                                                       make_float4(osc[0], osc[1], osc[2], 0.f), out, f->N);
    return check_launch("project");
}

pfgb_status ensure_train(pfgb_fno *f) {
    if (f->train) return PFGB_OK;
    const size_t act = (size_t)kW * f->N;
    f->vs.assign(f->L + 1, nullptr);
    f->pres.assign(f->L, nullptr);
    f->Cs.assign(f->L, nullptr);
    for (int l = 0; l <= f->L; ++l) FNO_CHECK(fno_alloc_t(f, &f->vs[l], act));
    for (int l = 0; l < f->L; ++l) {
        FNO_CHECK(fno_alloc_t(f, &f->pres[l], act));
        FNO_CHECK(fno_alloc_t(f, &f->Cs[l], (size_t)kW * f->M));
    }
    for (int i = 0; i < 3; ++i) FNO_CHECK(fno_alloc_t(f, &f->G[i], act));
    FNO_CHECK(fno_alloc_t(f, &f->grad, (size_t)f->nparams));
    FNO_CHECK(fno_alloc_t(f, &f->am, (size_t)f->nparams));
    FNO_CHECK(fno_alloc_t(f, &f->av, (size_t)f->nparams));
    FNO_TRY(cudaMemsetAsync(f->grad, 0, sizeof(float) * f->nparams, f->stream));
    FNO_TRY(cudaMemsetAsync(f->am, 0, sizeof(float) * f->nparams, f->stream));
    FNO_TRY(cudaMemsetAsync(f->av, 0, sizeof(float) * f->nparams, f->stream));
    FNO_CHECK(fno_alloc_t(f, &f->part, (size_t)kRedBlocks * kProjE));
    FNO_CHECK(fno_alloc_t(f, &f->dpart, (size_t)4 * kRedBlocks));
    f->train = true;
    return PFGB_OK;
}

pfgb_status reduce_into(pfgb_fno *f, int nb, int E, long long off, int accumulate) {
    k_reduce_part<<<(E + 31) / 32, 1024, 0, f->stream>>>(f->part, nb, E, f->grad + off, accumulate);
    return check_launch("reduce_part");
}

pfgb_status loss_grad_impl(pfgb_fno *f, const float *in, const float *tgt, int accumulate) {
    FNO_CHECK(ensure_train(f));
    FNO_CHECK(forward_impl(f, in, nullptr, true));
    const long long nt = 3 * f->N;
    const int nbs = 4 * 152;
    double *den = f->dscal, *loss = f->dscal + 1;
    k_sumsq<<<nbs, 256, 0, f->stream>>>(tgt, nt, f->dpart);
    FNO_CHECK(check_launch("sumsq"));
    k_sum_partials<<<1, 256, 0, f->stream>>>(f->dpart, nbs, den);
    FNO_CHECK(check_launch("sum_partials"));
    const long long ntiles = (f->N + kTile - 1) / kTile;
    const int nb = (int)std::min<long long>(ntiles, kRedBlocks);
    const float *osc = f->cfg.out_scale, *is = f->cfg.in_scale;
    const size_t sp = sizeof(float) * project_bwd_smem_floats();
    FNO_CHECK(smem_opt_in(k_project_bwd, sp));
    float *ga = f->G[0], *gp = f->G[1], *gc = f->G[2];
    k_project_bwd<<<nb, kTile, sp, f->stream>>>(f->vs[f->L], tgt, f->wbf + f->offQ1, f->master + f->offq1,
                                                f->wbf + f->offQ2, f->master + f->offq2,
                                                make_float4(osc[0], osc[1], osc[2], 0.f), den, ga, f->part,
                                                f->dpart + kRedBlocks, f->N, ntiles);
    FNO_CHECK(check_launch("project_bwd"));
    FNO_CHECK(reduce_into(f, nb, kProjE, f->offQ1, accumulate));
    k_loss_final<<<1, 256, 0, f->stream>>>(f->dpart + kRedBlocks, nb, den, loss);
    FNO_CHECK(check_launch("loss_final"));
    const float invN = (float)(1.0 / (double)f->N);
    const int LBz = lines_per_block(f->Z);
    const size_t sc = sizeof(float2) * ((size_t)f->Mz * f->Z + (size_t)kW * LBz * f->Mz);
    FNO_CHECK(smem_opt_in(k_idft_z_acc, sc));
    for (int l = f->L - 1; l >= 0; --l) {
        if (l == f->L - 1)
            k_layer_bwd<true><<<nb, kTile, 0, f->stream>>>(ga, f->pres[l], f->vs[l], f->wbf + f->offW[l], gp, gc,
                                                          f->part, f->N, ntiles);
        else
            k_layer_bwd<false><<<nb, kTile, 0, f->stream>>>(ga, f->pres[l], f->vs[l], f->wbf + f->offW[l], gp, gc,
                                                           f->part, f->N, ntiles);
        FNO_CHECK(check_launch("layer_bwd"));
        FNO_CHECK(reduce_into(f, nb, kLayerE, f->offW[l], accumulate));
        // adjoint of the inverse z (c2r weights 1, 2, 2, ...), then y and x onto the modes
        FNO_CHECK(spec_forward(f, gp, f->O, 1.f, 2.f));
        const long long nr = (long long)kW * kW * f->M;
        k_mode_grad<<<(unsigned)((nr + 255) / 256), 256, 0, f->stream>>>(
            f->Cs[l], f->O, reinterpret_cast<float2 *>(f->grad + f->offR[l]), (int)f->M, accumulate);
        FNO_CHECK(check_launch("mode_grad"));
        const long long nm = (long long)kW * f->M;
        k_mode_mix_adj<<<(unsigned)((nm + 255) / 256), 256, 0, f->stream>>>(
            f->O, reinterpret_cast<const __nv_bfloat162 *>(f->wbf + f->offR[l]), f->C, (int)f->M);
        FNO_CHECK(check_launch("mode_mix_adj"));
        FNO_CHECK(spec_inverse_xy(f, f->C));
        k_idft_z_acc<<<(unsigned)((f->S + LBz - 1) / LBz), 256, sc, f->stream>>>(f->A, gc, f->gz, f->S, f->Z,
                                                                                f->Mz, LBz, invN, invN);
        FNO_CHECK(check_launch("idft_z_acc"));
        std::swap(ga, gc);
    }
    const float4 s03 = make_float4(is[0], is[1], is[2], is[3]), s47 = make_float4(is[4], is[5], is[6], is[7]);
    k_lift_bwd<<<nb, kTile, 0, f->stream>>>(ga, in, s03, s47, f->part, f->N, ntiles);
    FNO_CHECK(check_launch("lift_bwd"));
    return reduce_into(f, nb, kLiftE, f->offP, accumulate);
}

void fno_free(pfgb_fno *f) {
    if (!f) return;
    if (f->stream) cudaStreamSynchronize(f->stream);
    else cudaDeviceSynchronize();
    for (void *p : f->allocs) cudaFree(p);
    delete f;
}

pfgb_status create_impl(const pfgb_fno_config *cfg, int device, const float *params, pfgb_fno **out) {
    FNO_CHECK(validate(cfg));
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        pfgb_set_error_msg("FNO: no CUDA device");
        return PFGB_ERR_CUDA;
    }
    if (device < 0 || device >= ndev) {
        pfgb_set_error_msg("FNO: device %d outside [0, %d)", device, ndev);
        return PFGB_ERR_INVALID;
    }
    FNO_TRY(cudaSetDevice(device));
    pfgb_fno *f = new pfgb_fno();
    f->cfg = *cfg;
    f->device = device;
    f->X = cfg->Nx; f->Y = cfg->Ny; f->Z = cfg->Nz; f->m = cfg->modes; f->L = cfg->layers;
    f->Mz = f->m;
    f->Q = 2 * f->m * f->Mz;
    f->N = (long long)f->X * f->Y * f->Z;
    f->S = (long long)f->X * f->Y;
    f->M = 4LL * f->m * f->m * f->m;
    layout_offsets(f);
    auto fail = [&](pfgb_status s) { fno_free(f); return s; };
    pfgb_status s;
    if ((s = upload_tw(f, &f->twx, f->X)) != PFGB_OK) return fail(s);
    if ((s = upload_tw(f, &f->twy, f->Y)) != PFGB_OK) return fail(s);
    {
        std::vector<float2> h((size_t)2 * f->m * f->Y);
        for (int j = 0; j < 2 * f->m; ++j) {
            const long long ky = j < f->m ? j : f->Y - 2 * f->m + j;
            for (int y = 0; y < f->Y; ++y) {
                const double a = 2.0 * PFGB_PI * (double)((ky * y) % f->Y) / (double)f->Y;
                h[(size_t)j * f->Y + y] = make_float2((float)cos(a), (float)sin(a));
            }
        }
        if ((s = fno_alloc_t(f, &f->tyi, h.size())) != PFGB_OK) return fail(s);
        if (cudaMemcpy(f->tyi, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
            pfgb_set_error_msg("FNO: twiddle upload failed");
            return fail(PFGB_ERR_CUDA);
        }
        const int M2 = pad2(f->Mz);
        std::vector<float2> hf((size_t)f->Z * M2), hg((size_t)f->Mz * f->Z);
        for (int z = 0; z < f->Z; ++z)
            for (int k = 0; k < M2; ++k) {
                const double a = -2.0 * PFGB_PI * (double)(((long long)k * z) % f->Z) / (double)f->Z;
                const float2 t = make_float2((float)cos(a), (float)sin(a));
                hf[(size_t)z * M2 + k] = k < f->Mz ? t : make_float2(0.f, 0.f);
                if (k < f->Mz) hg[(size_t)k * f->Z + z] = t;
            }
        if ((s = fno_alloc_t(f, &f->fz, hf.size() / 2)) != PFGB_OK) return fail(s);
        if ((s = fno_alloc_t(f, &f->gz, hg.size())) != PFGB_OK) return fail(s);
        if (cudaMemcpy(f->fz, hf.data(), sizeof(float2) * hf.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(f->gz, hg.data(), sizeof(float2) * hg.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
            pfgb_set_error_msg("FNO: twiddle upload failed");
            return fail(PFGB_ERR_CUDA);
        }
    }
    if ((s = fno_alloc_t(f, &f->master, (size_t)f->nparams)) != PFGB_OK) return fail(s);
    if ((s = fno_alloc_t(f, &f->wbf, (size_t)f->nparams)) != PFGB_OK) return fail(s);
    const size_t act = (size_t)kW * f->N;
    if ((s = fno_alloc_t(f, &f->va, act)) != PFGB_OK) return fail(s);
    if ((s = fno_alloc_t(f, &f->vb, act)) != PFGB_OK) return fail(s);
    if ((s = fno_alloc_t(f, &f->A, (size_t)kW * f->S * f->Mz)) != PFGB_OK) return fail(s);
    if ((s = fno_alloc_t(f, &f->B, (size_t)kW * f->X * f->Q)) != PFGB_OK) return fail(s);
    if ((s = fno_alloc_t(f, &f->C, (size_t)kW * f->M)) != PFGB_OK) return fail(s);
    if ((s = fno_alloc_t(f, &f->O, (size_t)kW * f->M)) != PFGB_OK) return fail(s);
    if ((s = fno_alloc_t(f, &f->dscal, 8)) != PFGB_OK) return fail(s);
    std::vector<float> h;
    if (params) h.assign(params, params + f->nparams);
    else init_params(f, h);
    if (cudaMemcpy(f->master, h.data(), sizeof(float) * f->nparams, cudaMemcpyHostToDevice) != cudaSuccess) {
        pfgb_set_error_msg("FNO: parameter upload failed");
        return fail(PFGB_ERR_CUDA);
    }
    k_to_bf16<<<1216, 256>>>(f->master, f->wbf, f->nparams);
    if (cudaDeviceSynchronize() != cudaSuccess || cudaGetLastError() != cudaSuccess) {
        pfgb_set_error_msg("FNO: weight conversion failed");
        return fail(PFGB_ERR_CUDA);
    }
    *out = f;
    return PFGB_OK;
}

const char kMagic[8] = {'P', 'F', 'G', 'B', 'F', 'N', 'O', '1'};

}  // namespace

int pfgb_fno_device(const pfgb_fno *f) { return f ? f->device : -1; }
long long pfgb_fno_forward_launches(const pfgb_fno *f) { return f ? 2 + 7LL * f->L : 0; }

extern "C" {

void pfgb_fno_config_default(pfgb_fno_config *c) {
    if (!c) return;
    std::memset(c, 0, sizeof(*c));
    c->Nx = c->Ny = c->Nz = 128;
    c->modes = 12;
    c->layers = 4;
    c->seed = 20240611ull;
    for (int i = 0; i < kIn; ++i) c->in_scale[i] = 1.f;
    for (int i = 0; i < kOut; ++i) c->out_scale[i] = 1.f;
}

pfgb_status pfgb_fno_create(const pfgb_fno_config *cfg, int device, pfgb_fno **out) {
    if (!cfg || !out) return PFGB_ERR_INVALID;
    *out = nullptr;
    return create_impl(cfg, device, nullptr, out);
}

void pfgb_fno_destroy(pfgb_fno *f) { fno_free(f); }

pfgb_status pfgb_fno_set_stream(pfgb_fno *f, void *stream) {
    if (!f) return PFGB_ERR_INVALID;
    if (f->stream != (cudaStream_t)stream) FNO_TRY(cudaStreamSynchronize(f->stream));
    f->stream = (cudaStream_t)stream;
    return PFGB_OK;
}

long long pfgb_fno_num_params(const pfgb_fno *f) { return f ? f->nparams : -1; }

pfgb_status pfgb_fno_get_config(const pfgb_fno *f, pfgb_fno_config *cfg) {
    if (!f || !cfg) return PFGB_ERR_INVALID;
    *cfg = f->cfg;
    return PFGB_OK;
}

pfgb_status pfgb_fno_set_scales(pfgb_fno *f, const float *in_scale, const float *out_scale) {
    if (!f) return PFGB_ERR_INVALID;
    pfgb_fno_config c = f->cfg;
    if (in_scale) std::memcpy(c.in_scale, in_scale, sizeof(c.in_scale));
    if (out_scale) std::memcpy(c.out_scale, out_scale, sizeof(c.out_scale));
    FNO_CHECK(validate(&c));
    f->cfg = c;
    return PFGB_OK;
}

pfgb_status pfgb_fno_get_params(pfgb_fno *f, float *host, long long n) {
    if (!f || !host || n != f->nparams) {
        pfgb_set_error_msg("FNO: get_params wants %lld floats", f ? f->nparams : -1LL);
        return PFGB_ERR_INVALID;
    }
    FNO_TRY(cudaSetDevice(f->device));
    FNO_TRY(cudaMemcpyAsync(host, f->master, sizeof(float) * n, cudaMemcpyDeviceToHost, f->stream));
    FNO_TRY(cudaStreamSynchronize(f->stream));
    return PFGB_OK;
}

pfgb_status pfgb_fno_set_params(pfgb_fno *f, const float *host, long long n) {
    if (!f || !host || n != f->nparams) {
        pfgb_set_error_msg("FNO: set_params wants %lld floats", f ? f->nparams : -1LL);
        return PFGB_ERR_INVALID;
    }
    FNO_TRY(cudaSetDevice(f->device));
    FNO_TRY(cudaMemcpyAsync(f->master, host, sizeof(float) * n, cudaMemcpyHostToDevice, f->stream));
    k_to_bf16<<<1216, 256, 0, f->stream>>>(f->master, f->wbf, f->nparams);
    FNO_CHECK(check_launch("to_bf16"));
    if (f->train) {
        FNO_TRY(cudaMemsetAsync(f->am, 0, sizeof(float) * f->nparams, f->stream));
        FNO_TRY(cudaMemsetAsync(f->av, 0, sizeof(float) * f->nparams, f->stream));
    }
    f->adam_t = 0;
    FNO_TRY(cudaStreamSynchronize(f->stream));
    return PFGB_OK;
}

pfgb_status pfgb_fno_forward(pfgb_fno *f, const float *d_in, float *d_out) {
    if (!f || !d_in || !d_out) return PFGB_ERR_INVALID;
    FNO_TRY(cudaSetDevice(f->device));
    return forward_impl(f, d_in, d_out, false);
}

pfgb_status pfgb_fno_loss_grad(pfgb_fno *f, const float *d_in, const float *d_target, int accumulate,
                               double *loss) {
    if (!f || !d_in || !d_target) return PFGB_ERR_INVALID;
    FNO_TRY(cudaSetDevice(f->device));
    FNO_CHECK(loss_grad_impl(f, d_in, d_target, accumulate));
    if (loss) {
        FNO_TRY(cudaMemcpyAsync(loss, f->dscal + 1, sizeof(double), cudaMemcpyDeviceToHost, f->stream));
        FNO_TRY(cudaStreamSynchronize(f->stream));
        if (!std::isfinite(*loss)) {
            pfgb_set_error_msg("FNO: non-finite loss");
            return PFGB_ERR_NONFINITE;
        }
    }
    return PFGB_OK;
}

pfgb_status pfgb_fno_get_grad(pfgb_fno *f, float *host, long long n) {
    if (!f || !host || n != f->nparams || !f->train) {
        pfgb_set_error_msg("FNO: get_grad wants %lld floats after a loss_grad call", f ? f->nparams : -1LL);
        return PFGB_ERR_INVALID;
    }
    FNO_TRY(cudaSetDevice(f->device));
    FNO_TRY(cudaMemcpyAsync(host, f->grad, sizeof(float) * n, cudaMemcpyDeviceToHost, f->stream));
    FNO_TRY(cudaStreamSynchronize(f->stream));
    return PFGB_OK;
}

pfgb_status pfgb_fno_adam_step(pfgb_fno *f, const pfgb_fno_adam *opt) {
    if (!f || !opt || !f->train) {
        pfgb_set_error_msg("FNO: adam_step needs an optimizer and a loss_grad call first");
        return PFGB_ERR_INVALID;
    }
    if (!(opt->lr >= 0.f) || !(opt->beta1 >= 0.f && opt->beta1 < 1.f) || !(opt->beta2 >= 0.f && opt->beta2 < 1.f) ||
        !(opt->eps > 0.f)) {
        pfgb_set_error_msg("FNO: invalid Adam hyper-parameters");
        return PFGB_ERR_INVALID;
    }
    FNO_TRY(cudaSetDevice(f->device));
    f->adam_t++;
    const float bc1 = (float)(1.0 - pow((double)opt->beta1, (double)f->adam_t));
    const float bc2 = (float)(1.0 - pow((double)opt->beta2, (double)f->adam_t));
    double *gn = f->dscal + 2;
    if (opt->clip_norm > 0.f) {
        k_sumsq_f<<<4 * 152, 256, 0, f->stream>>>(f->grad, f->nparams, f->dpart);
        FNO_CHECK(check_launch("grad_norm"));
        k_sum_partials<<<1, 256, 0, f->stream>>>(f->dpart, 4 * 152, gn);
        FNO_CHECK(check_launch("grad_norm_sum"));
    }
    k_adam<<<1216, 256, 0, f->stream>>>(f->master, f->wbf, f->grad, f->am, f->av, f->nparams, opt->lr, opt->beta1,
                                        opt->beta2, opt->eps, opt->weight_decay, bc1, bc2, opt->clip_norm, gn);
    return check_launch("adam");
}

pfgb_status pfgb_fno_save(pfgb_fno *f, const char *path) {
    if (!f || !path) return PFGB_ERR_INVALID;
    std::vector<float> h((size_t)f->nparams);
    FNO_CHECK(pfgb_fno_get_params(f, h.data(), f->nparams));
    FILE *fp = fopen(path, "wb");
    if (!fp) { pfgb_set_error_msg("FNO: cannot write %s", path); return PFGB_ERR_IO; }
    int32_t hdr[10] = {1, f->cfg.Nx, f->cfg.Ny, f->cfg.Nz, f->cfg.modes, f->cfg.layers, kW, kH, kIn, kOut};
    const long long n = f->nparams;
    bool ok = fwrite(kMagic, 1, 8, fp) == 8 && fwrite(hdr, sizeof(hdr), 1, fp) == 1 &&
              fwrite(f->cfg.in_scale, sizeof(float), kIn, fp) == (size_t)kIn &&
              fwrite(f->cfg.out_scale, sizeof(float), kOut, fp) == (size_t)kOut &&
              fwrite(&n, sizeof(n), 1, fp) == 1 && fwrite(h.data(), sizeof(float), h.size(), fp) == h.size();
    ok = (fclose(fp) == 0) && ok;
    if (!ok) { pfgb_set_error_msg("FNO: short write to %s", path); return PFGB_ERR_IO; }
    return PFGB_OK;
}

pfgb_status pfgb_fno_load(const char *path, int Nx, int Ny, int Nz, int device, pfgb_fno **out) {
    if (!path || !out) return PFGB_ERR_INVALID;
    *out = nullptr;
    FILE *fp = fopen(path, "rb");
    if (!fp) { pfgb_set_error_msg("FNO: cannot read %s", path); return PFGB_ERR_IO; }
    char mg[8];
    int32_t hdr[10];
    pfgb_fno_config c;
    pfgb_fno_config_default(&c);
    long long n = 0;
    bool ok = fread(mg, 1, 8, fp) == 8 && std::memcmp(mg, kMagic, 8) == 0 && fread(hdr, sizeof(hdr), 1, fp) == 1 &&
              hdr[0] == 1 && hdr[6] == kW && hdr[7] == kH && hdr[8] == kIn && hdr[9] == kOut &&
              fread(c.in_scale, sizeof(float), kIn, fp) == (size_t)kIn &&
              fread(c.out_scale, sizeof(float), kOut, fp) == (size_t)kOut && fread(&n, sizeof(n), 1, fp) == 1;
    std::vector<float> h;
    if (ok) {
        c.Nx = Nx > 0 ? Nx : hdr[1];
        c.Ny = Ny > 0 ? Ny : hdr[2];
        c.Nz = Nz > 0 ? Nz : hdr[3];
        c.modes = hdr[4];
        c.layers = hdr[5];
        const long long expect = (long long)kW * kIn + kW +
                                 (long long)c.layers * (kW * kW + kW + 2LL * kW * kW * 4LL * c.modes * c.modes * c.modes) +
                                 kH * kW + kH + kOut * kH + kOut;
        ok = n == expect;
        if (ok) {
            h.resize((size_t)n);
            ok = fread(h.data(), sizeof(float), h.size(), fp) == h.size();
        }
    }
    fclose(fp);
    if (!ok) { pfgb_set_error_msg("FNO: %s is not a model file of this library", path); return PFGB_ERR_IO; }
    return create_impl(&c, device, h.data(), out);
}

}  // extern "C"
