"""The product of a double h with floats on the FP32 pipe (physics.cuh): h is not
rounded to float first."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "physics.cuh"
template <typename T> __global__ void k(const double *h, const float *w, const float *s, float *o, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) o[i] = h_scaled<T, float>((T)h[i], w[i], s[i]);
}
extern "C" int run(int fp64, const double *h, const float *w, const float *s, float *o, int n) {
    if (fp64) k<double><<<(n + 255) / 256, 256>>>(h, w, s, o, n);
    else k<float><<<(n + 255) / 256, 256>>>(h, w, s, o, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.mark.parametrize("fp64", [1, 0])
def test_h_scaled(tmp_path, fp64):
    """FP64 fields: two roundings, of w s and of the product with h; FP32 fields:
    (h w) s as floats."""
    import torch
    from cuda_sto_pf_gb300 import build
    (tmp_path / "h.cu").write_text(SRC)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-I", build.CSRC, "-shared", "-o", str(tmp_path / "h.so"),
                    str(tmp_path / "h.cu")], check=True)
    rng = np.random.default_rng(3)
    n = 1 << 16
    h = rng.uniform(-1.0, 2.0, n) * 10.0 ** rng.integers(-6, 1, n)
    w, s = (rng.uniform(-1.0, 1.0, n).astype(np.float32) for _ in range(2))
    d = [torch.from_numpy(x).cuda() for x in (h, w, s)] + [torch.empty(n, dtype=torch.float32, device="cuda")]
    torch.cuda.synchronize()
    assert ctypes.CDLL(str(tmp_path / "h.so")).run(fp64, *[ctypes.c_void_p(x.data_ptr()) for x in d], n) == 0
    got = d[3].cpu().numpy()
    if fp64:
        want = h * (w * s).astype(np.float64)      # w s rounded to float, then exact to 53 bits
        assert (np.abs(got - want) <= 2.0 ** -24 * (1 + 2.0 ** -20) * np.abs(want)).all()
    else:
        assert np.array_equal(got, h.astype(np.float32) * w * s)
