"""FP32 butterflies with irrational or half factors (fft.cuh): a product goes into its
sum with one rounding."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "fft.cuh"
template <int R, int DIR> __global__ void k(const float2 *in, float2 *out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 v[R];
    for (int r = 0; r < R; ++r) v[r] = in[i * R + r];
    if constexpr (R == 3) bfly3<float, DIR>(v);
    else if constexpr (R == 5) bfly5<float, DIR>(v);
    else if constexpr (R == 6) bfly6<float, DIR>(v);
    else bfly8<float, DIR>(v);
    for (int r = 0; r < R; ++r) out[i * R + r] = v[r];
}
template <int DIR> static int go(int R, const float2 *in, float2 *out, int n) {
    const int b = (n + 255) / 256;
    if (R == 3) k<3, DIR><<<b, 256>>>(in, out, n);
    else if (R == 5) k<5, DIR><<<b, 256>>>(in, out, n);
    else if (R == 6) k<6, DIR><<<b, 256>>>(in, out, n);
    else k<8, DIR><<<b, 256>>>(in, out, n);
    return (int)cudaDeviceSynchronize();
}
extern "C" int run(int R, int dir, const float2 *in, float2 *out, int n) {
    return dir < 0 ? go<-1>(R, in, out, n) : go<1>(R, in, out, n);
}
"""
S3, R2 = np.float32(np.sqrt(0.75)), np.float32(np.sqrt(0.5))
C1, C2 = np.float32(0.25 * (np.sqrt(5) - 1)), np.float32(-0.25 * (np.sqrt(5) + 1))
S1, S2 = np.float32(np.sin(0.4 * np.pi)), np.float32(np.sin(0.8 * np.pi))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from cuda_sto_pf_gb300 import build
    d = tmp_path_factory.mktemp("bf")
    (d / "bf.cu").write_text(SRC)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-I", build.CSRC, "-shared", "-o", str(d / "bf.so"), str(d / "bf.cu")],
                   check=True)
    return ctypes.CDLL(str(d / "bf.so"))


def _r(z):
    """one rounding to float of both parts"""
    return z.astype(np.complex64).astype(np.complex128)


def _mad(a, k, b):
    """k a + b, exact but for one rounding (the product is exact in a double)"""
    return _r(a * np.float64(k) + b)


def _b3(v, rot):
    s, d = _r(v[1] + v[2]), _r(v[1] - v[2])
    m = _mad(s, -0.5, v[0])
    return [_r(v[0] + s), _mad(rot * d, S3, m), _mad(rot * d, -S3, m)]


def _b4(v, rot):
    t0, t1, t2, t3 = _r(v[0] + v[2]), _r(v[0] - v[2]), _r(v[1] + v[3]), rot * _r(v[1] - v[3])
    return [_r(t0 + t2), _r(t1 + t3), _r(t0 - t2), _r(t1 - t3)]


def _want(R, v, rot):
    if R == 3:
        return _b3(v, rot)
    if R == 5:
        a1, b1, a2, b2 = _r(v[1] + v[4]), _r(v[1] - v[4]), _r(v[2] + v[3]), _r(v[2] - v[3])
        p1, p2 = _mad(a2, C2, _mad(a1, C1, v[0])), _mad(a2, C1, _mad(a1, C2, v[0]))
        b1, b2 = rot * b1, rot * b2
        return [_r(_r(v[0] + a1) + a2), _mad(b1, S1, _mad(b2, S2, p1)), _mad(b1, S2, _mad(b2, -S1, p2)),
                _mad(b1, -S2, _mad(b2, S1, p2)), _mad(b1, -S1, _mad(b2, -S2, p1))]
    if R == 6:
        e, o = _b3(v[0::2], rot), _b3(v[1::2], rot)
        f = [lambda s: _r(e[0] + s * o[0]), lambda s: _mad(o[1], 0.5 * s, _mad(rot * o[1], S3 * np.float32(s), e[1])),
             lambda s: _mad(o[2], -0.5 * s, _mad(rot * o[2], S3 * np.float32(s), e[2]))]
        return [g(1) for g in f] + [g(-1) for g in f]
    e, o = _b4(v[0::2], rot), _b4(v[1::2], rot)
    t1, t3 = _r(o[1] + rot * o[1]), _r(rot * o[3] - o[3])
    f = [lambda s: _r(e[0] + s * o[0]), lambda s: _mad(t1, R2 * np.float32(s), e[1]), lambda s: _r(e[2] + s * (rot * o[2])),
         lambda s: _mad(t3, R2 * np.float32(s), e[3])]
    return [g(1) for g in f] + [g(-1) for g in f]


@pytest.mark.parametrize("direction", [-1, 1])
@pytest.mark.parametrize("R", [3, 5, 6, 8])
def test_products_are_fused(lib, R, direction):
    """Bit for bit but where the double sum of product and summand rounds to a tie
    (one value in some 2^28)."""
    import torch
    n = 1 << 14
    rng = np.random.default_rng(R)
    x = (rng.standard_normal((n, R)) + 1j * rng.standard_normal((n, R))).astype(np.complex64)
    d = torch.from_numpy(x).cuda()
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    assert lib.run(R, direction, ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(out.data_ptr()), n) == 0
    got = out.cpu().numpy()
    want = np.stack(_want(R, list(x.T.astype(np.complex128)), 1j * direction), axis=1).astype(np.complex64)
    assert (got != want).sum() <= 2
    exact = np.fft.fft(x.astype(np.complex128)) if direction < 0 else np.fft.ifft(x.astype(np.complex128)) * R
    assert np.abs(got - exact).max() <= 1e-6 * np.abs(exact).max()
