"""Sums of floats and of their squares on the FP32 pipe (fsum, dfloat.cuh) against
exactly rounded sums: no further off than float64 sums are, over a float's whole
range."""
import ctypes
import math
import subprocess
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one block; its threads' sums are merged as the solver's block reductions do
SRC = r"""
#include "dfloat.cuh"
template <int KIND> __global__ void k_sum(const float *v, const float *q, const float *w, int n, double *out) {
    __shared__ fsum red[32];
    fsum s = fs_zero();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        if (KIND == 3) {
            if (!fs_add_product(s, w[i], df_two_sum(v[i], -q[i]))) s.x += (double)w[i] * ((double)v[i] - (double)q[i]);
        } else if (KIND == 2) fs_add_square_diff(s, v[i], q[i]);
        else KIND ? fs_add_square(s, v[i]) : fs_add(s, v[i]);
    }
    for (int o = 16; o > 0; o >>= 1) fs_merge(s, fs_shfl_down(s, o));
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)blockDim.x / 32; ++w) fs_merge(s, red[w]);
        out[0] = fs_to_double(s);
    }
}
extern "C" int run(int kind, const float *v, const float *q, const float *w, int n, double *out) {
    if (kind == 3) k_sum<3><<<1, 256>>>(v, q, w, n, out);
    else if (kind == 2) k_sum<2><<<1, 256>>>(v, q, w, n, out);
    else if (kind) k_sum<1><<<1, 256>>>(v, q, w, n, out);
    else k_sum<0><<<1, 256>>>(v, q, w, n, out);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from cuda_sto_pf_gb300 import build
    d = tmp_path_factory.mktemp("fs")
    (d / "fs.cu").write_text(SRC)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-I", build.CSRC, "-shared", "-o", str(d / "fs.so"), str(d / "fs.cu")],
                   check=True)
    return ctypes.CDLL(str(d / "fs.so"))


def _sum(lib, v, square, q=None, w=None):
    import torch
    d = [torch.from_numpy(np.ascontiguousarray(v if x is None else x, dtype=np.float32)).cuda() for x in (v, q, w)]
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(x.data_ptr()) for x in (*d, out)]
    kind = 3 if w is not None else 2 if q is not None else int(square)
    assert lib.run(kind, p[0], p[1], p[2], v.size, p[3]) == 0
    return out.item()


def _values(kind, n):
    rng = np.random.default_rng(n)
    u = rng.uniform(-1.0, 1.0, n)
    return {"near": np.abs(u) + 0.25, "signed": u, "wide": u * 10.0 ** rng.uniform(-12, 12, n),
            "small": u * 1e-24, "tiny": u * 1e-38, "large": np.abs(u) * 1e30, "huge": np.abs(u) * 3e38,
            "zeros": 0.0 * u, "mixed": u * 10.0 ** rng.uniform(-37, 38, n)}[kind].astype(np.float32)


@pytest.mark.parametrize("square", [False, True])
@pytest.mark.parametrize("n", [1, 255, 100003])
@pytest.mark.parametrize("kind", ["near", "signed", "wide", "small", "tiny", "large", "huge", "zeros", "mixed"])
def test_sums_hold_float64_precision(lib, kind, n, square):
    """Within 2^-53 of the sum of magnitudes for each rounding to float64: three in
    the final conversion (and the compensated sum's own error, below one), and
    where values are beyond its range, a thread's terms with their squares and
    twelve merges, as in a plain float64 sum."""
    v = _values(kind, n)
    a = np.abs(v.astype(np.float64))
    t = (v.astype(np.float64) ** 2 if square else v.astype(np.float64)).tolist()
    beyond = ((a != 0) & ((a <= 2.0 ** -46) | (a >= 2.0 ** 48))).any() if square else (a >= 2.0 ** 96).any()
    roundings = 4 + (math.ceil(n / 256) + 13 if beyond else 0)
    assert abs(_sum(lib, v, square) - math.fsum(t)) <= 2.0 ** -53 * roundings * math.fsum(map(abs, t))


@pytest.mark.parametrize("square", [False, True])
def test_infinities_and_nan_reach_the_sum(lib, square):
    v = np.ones(300, dtype=np.float32)
    v[200] = np.inf
    assert _sum(lib, v, square) == math.inf
    v[17] = np.nan
    assert math.isnan(_sum(lib, v, square))


@pytest.mark.parametrize("step", [0.0, 1e-9, 1e-3, 0.7])
def test_squared_differences(lib, step):
    """Squares of differences, exact in a float or not: two roundings to float64 a
    term where they are not, a thread's terms and twelve merges."""
    rng = np.random.default_rng(8)
    p = (rng.uniform(0.0, 1.0, 4099) ** 8).astype(np.float32)
    q = np.clip(p + step * rng.uniform(-1.0, 1.0, p.size), 0.0, 1.0).astype(np.float32)
    t = ((p.astype(np.float64) - q.astype(np.float64)) ** 2).tolist()
    want = math.fsum(t)
    assert abs(_sum(lib, p, True, q) - want) <= 2.0 ** -53 * (math.ceil(p.size / 256) + 19) * want


@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e-11, 1e-30, 1e20])
def test_products_with_differences(lib, scale):
    """a (p - q), exact in the sum over the range of its products; two roundings to
    float64 a term beyond it."""
    rng = np.random.default_rng(9)
    n = 4099
    a = (rng.uniform(-1.0, 1.0, n) * 10.0 ** rng.uniform(-3, 3, n)).astype(np.float32)
    p = (scale * rng.uniform(-1.0, 1.0, n)).astype(np.float32)
    q = (scale * rng.uniform(-1.0, 1.0, n) * 10.0 ** rng.uniform(-6, 0, n)).astype(np.float32)
    t = [Fraction(float(x)) * (Fraction(float(y)) - Fraction(float(z))) for x, y, z in zip(a, p, q)]
    mag = float(sum(map(abs, t)))
    err = float(abs(Fraction(_sum(lib, p, False, q, a)) - sum(t)))
    roundings = 5 if 1e-9 < scale < 1e9 else math.ceil(n / 256) + 19
    assert err <= 2.0 ** -53 * roundings * mag
