"""The stages that a line transform is planned in (fft.cuh), for every length the
entry points take: what each stage of fftline.cu relies on holds, and the
stages' index arithmetic gives the discrete Fourier transform.  On a GPU, the
lengths whose smallest radix would leave the last stage more butterflies than a
block has threads."""
import json
import subprocess

import numpy as np
import pytest

from test_gpu_fft import _run

# prints one plan per line: n, its stages, and the least and the largest number
# of threads over every count of lines that a tile can have
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include "fft.cuh"
static int g_news = 0;
__host__ __device__ void *operator new(size_t n) {
#ifndef __CUDA_ARCH__
    ++g_news;
#endif
    return malloc(n);
}
__host__ __device__ void operator delete(void *p) noexcept { free(p); }
__host__ __device__ void operator delete(void *p, size_t) noexcept { free(p); }
int main() {
    for (int n = 1; n <= PFGB_MAX_N; ++n) {
        AxisPlan p;
        const int before = g_news;
        const bool ok = pfgb_make_plan(n, &p);
        const int news = g_news - before;
        std::printf("{\"n\": %d, \"ok\": %s, \"news\": %d, \"stages\": [", n, ok ? "true" : "false", news);
        for (int s = 0; s < p.nst; ++s)
            std::printf("%s[%d, %d, %d, %d, %u, %u]", s ? ", " : "", p.st[s].R, p.st[s].B, p.st[s].m, p.st[s].kind,
                        p.st[s].fm.d, p.st[s].fR.d);
        int lo = 1 << 30, hi = 0;
        for (int L = 1; L <= 512; ++L) {
            const int t = pfgb_line_threads(p, L);
            lo = t < lo ? t : lo;
            hi = t > hi ? t : hi;
        }
        std::printf("], \"threads\": [%d, %d]}\n", lo, hi);
    }
}
"""
MAX_STAGES, DIRECT_SUMS = 16, 8


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    from cuda_sto_pf_gb300 import build
    d = tmp_path_factory.mktemp("plans")
    (d / "plans.cu").write_text(SRC)
    subprocess.run([build.NVCC, "-std=c++17", "-O1", "-I", build.CSRC, "-I", build.INCLUDE, "--expt-relaxed-constexpr",
                    *build.ARCH, "-o", str(d / "plans"), str(d / "plans.cu")], check=True)
    out = subprocess.run([str(d / "plans")], check=True, capture_output=True, text=True).stdout
    return [json.loads(l) for l in out.splitlines()]


def test_every_length_fits_its_stages(plans):
    """A last butterfly stage has a thread for each butterfly of a line, a direct
    stage the points of a line in eight sums per thread (a chunk of lines is
    blockDim / (n / R) and blockDim * 8 / n: never none), a 41-point stage comes
    first."""
    assert [p["n"] for p in plans] == list(range(1, 1025))
    for p in plans:
        n, st, (lo, hi) = p["n"], p["stages"], p["threads"]
        assert p["ok"] and len(st) <= MAX_STAGES and int(np.prod([s[0] for s in st])) == n, p
        assert 32 <= lo and hi <= 256 and lo % 32 == 0, p
        B = n
        for i, (R, b, m, kind, dm, dR) in enumerate(st):
            assert (b, m, dm, dR) == (B, B // R, B // R, R), p
            B = m
            if kind == 1:
                assert R == 41 and i == 0, p
            elif kind == 2:
                assert lo * DIRECT_SUMS // n >= 1, p
            else:
                assert kind == 0 and 2 <= R <= 16, p
                if i == len(st) - 1:
                    assert lo // (n // R) >= 1, p


def test_plans_allocate_nothing(plans):
    """They are made at C entries, one of which promises no allocation."""
    assert not any(p["news"] for p in plans)


def _emulate(x, stages):
    """The in-place stages of fftline.cu: each block's DFT of its R points, the
    twiddles, and the last stage's digit-reversed places."""
    n, v = x.size, x.astype(complex)
    for s, (R, B, m, kind, _, _) in enumerate(stages):
        last, nb, twst = s == len(stages) - 1, n // R, n // B
        j = np.arange(nb)
        b, jp = j // m, j % m
        r = np.arange(R)
        a = (b * B + jp)[:, None] + r * m
        W = np.exp(-2j * np.pi * np.outer(r, r) / R)
        y = (v[a] @ W) * np.exp(-2j * np.pi * ((jp[:, None] * r * twst) % n) / n)
        if not last or kind == 1:
            v[a] = y
            continue
        q, place = b.copy(), np.zeros_like(b)
        for t in range(len(stages) - 2, -1, -1):
            place = place * stages[t][0] + q % stages[t][0]
            q //= stages[t][0]
        v[place[:, None] + r * nb] = y
    return v


def test_stages_give_the_transform(plans):
    rng = np.random.default_rng(3)
    for p in plans:
        x = rng.standard_normal(p["n"]) + 1j * rng.standard_normal(p["n"])
        assert np.abs(_emulate(x, p["stages"]) - np.fft.fft(x)).max() <= 1e-12 * p["n"], p


# a direct prime (or two) and 2 or 3, and a smooth part whose largest radix is needed
# last, with and without Rader's 41
@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(0, 1e-13), (1, 3e-6)])
@pytest.mark.parametrize("n", [514, 578, 598, 774, 861, 902, 999, 1018, 1023])
def test_long_lengths_with_a_small_last_radix(capi, n, prec, tol):
    for shape in ((n, 3, 6), (2, n, 9), (5, 3, n)):
        x = np.random.default_rng(n).standard_normal(shape)
        k, back = _run(capi, prec, shape, x)
        ref = np.fft.rfftn(x)
        assert np.abs(k - ref).max() <= tol * np.abs(ref).max() * np.log2(x.size + 1), shape
        assert np.abs(back / x.size - x).max() <= tol * np.abs(x).max() * np.log2(x.size + 1), shape
