"""The double-float arithmetic of FP32 runs (dfloat.cuh) against float64: the
rounded quotients and products are the floats that the same expressions in
float64 round to, bit for bit, at ties of the rounding above all."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "dfloat.cuh"
__device__ dfl split(double v) { return df_from_double(v); }
__global__ void k_damped(const double *num, const double *m, const double *k2, float *out, int *ok, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ok[i] = df_round_damped(split(num[i]), split(m[i]), split(k2[i]), out + i);
}
__global__ void k_product(const double *a, const double *b, float *out, int *ok, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ok[i] = df_round_product(split(a[i]), split(b[i]), out + i);
}
extern "C" int run_damped(const double *num, const double *m, const double *k2, float *out, int *ok, int n) {
    k_damped<<<(n + 255) / 256, 256>>>(num, m, k2, out, ok, n);
    return (int)cudaDeviceSynchronize();
}
extern "C" int run_product(const double *a, const double *b, float *out, int *ok, int n) {
    k_product<<<(n + 255) / 256, 256>>>(a, b, out, ok, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from cuda_sto_pf_gb300 import build
    d = tmp_path_factory.mktemp("df")
    (d / "df.cu").write_text(SRC)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-I", build.CSRC, "-shared", "-o", str(d / "df.so"), str(d / "df.cu")],
                   check=True)
    return ctypes.CDLL(str(d / "df.so"))


def _call(f, *cols):
    import torch
    n = len(cols[0])
    d = [torch.from_numpy(np.ascontiguousarray(c, dtype=np.float64)).cuda() for c in cols]
    out = torch.empty(n, dtype=torch.float32, device="cuda")
    ok = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert f(*[ctypes.c_void_p(x.data_ptr()) for x in (*d, out, ok)], n) == 0
    return out.cpu().numpy(), ok.cpu().numpy() != 0


def _ties(rng, n):
    """doubles half way between two floats, and a few last places off"""
    f = rng.uniform(1.0, 2.0, n).astype(np.float32)
    t = 0.5 * (f.astype(np.float64) + np.nextafter(f, np.float32(4.0)).astype(np.float64))
    return t * (1.0 + rng.integers(-3, 4, n) * 2.0 ** -52)


def test_quotients_round_as_in_float64(lib):
    rng = np.random.default_rng(5)
    n = 1 << 18
    m, k2 = 10.0 ** rng.uniform(-12, 8, n), 10.0 ** rng.uniform(-3, 3, n)
    num = 10.0 ** rng.uniform(-10, 2, n)
    num[::2] = (_ties(rng, n) * (1.0 + m * k2))[::2] * 2.0 ** rng.integers(-30, 30, n)[::2]
    got, ok = _call(lib.run_damped, num, m, k2)
    want = (num / (1.0 + m * k2)).astype(np.float32)
    assert np.array_equal(got[ok], want[ok])
    assert ok[1::2].mean() > 0.999     # away from ties it decides


def test_products_round_as_in_float64(lib):
    rng = np.random.default_rng(6)
    n = 1 << 18
    a, b = 10.0 ** rng.uniform(-6, 6, n), 10.0 ** rng.uniform(-9, -2, n)
    a[::2] = (_ties(rng, n) / b)[::2]
    got, ok = _call(lib.run_product, a, b)
    assert np.array_equal(got[ok], (a * b).astype(np.float32)[ok])
    assert ok[1::2].mean() > 0.999


def test_what_leaves_the_range_is_not_decided(lib):
    big, tiny = 1e39, 1e-39
    rows = [(1.0, big, 1.0), (1.0, 1.0, big), (1.0, 1e20, 1e20), (1.0, -1.0, 1.0), (1.0, -0.75, 1.0), (np.inf, 1.0, 1.0),
            (np.nan, 1.0, 1.0), (1.0, np.nan, 1.0), (1.0, 1.0, np.inf), (big, 1.0, 1.0), (tiny, 1.0, 1.0), (0.0, 1.0, 1.0)]
    assert not _call(lib.run_damped, *map(list, zip(*rows)))[1].any()
    rows = [(big, 1.0), (tiny, 1.0), (0.0, 1.0), (np.inf, 1.0), (np.nan, 1.0), (1e30, 1e30), (1e-30, 1e-30)]
    assert not _call(lib.run_product, *map(list, zip(*rows)))[1].any()
