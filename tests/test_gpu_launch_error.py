"""A launch that the runtime refuses is reported by that launch and not left for
the thread's next call to find."""
import ctypes
import subprocess

import pytest

pytestmark = pytest.mark.gpu

# a block of 4096 threads: refused on the host, with nothing launched
SRC = r"""
#include "common.cuh"
void pfgb_set_error(const char *, cudaError_t, const char *, int) {}
void pfgb_set_error_msg(const char *, ...) {}
template <typename T> __global__ void k(int *) {}
extern "C" int run(int threads, int *left) {
    const cudaError_t e = pfgb_launch<float>(k<float>, dim3(1), dim3(threads), 0, nullptr, (int *)nullptr);
    *left = (int)cudaPeekAtLastError();
    cudaGetLastError();
    return (int)e;
}
"""


def test_refused_launch_leaves_no_error(tmp_path):
    import torch
    from cuda_sto_pf_gb300 import build
    torch.zeros(1, device="cuda")
    (tmp_path / "l.cu").write_text(SRC)
    subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-I", build.CSRC, "-shared", "-o", str(tmp_path / "l.so"),
                    str(tmp_path / "l.cu")], check=True)
    lib, left = ctypes.CDLL(str(tmp_path / "l.so")), ctypes.c_int(-1)
    assert lib.run(64, ctypes.byref(left)) == 0 and left.value == 0
    assert lib.run(4096, ctypes.byref(left)) != 0 and left.value == 0
    torch.cuda.synchronize()
