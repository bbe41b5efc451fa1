"""The line transforms' stages (fftline.cu) one by one, on the strided axes and
on z rows, against numpy at test_gpu_fft's tolerances."""
import numpy as np
import pytest

from test_gpu_fft import _run

pytestmark = pytest.mark.gpu

# one stage of every radix; each radix before a last stage and as one; three
# stages; Rader's 41 alone, first of two and of three; direct sums of one prime,
# of two, before and after a smooth part; the largest lengths
LENGTHS = [*range(2, 17), 17, 41, 47, 49, 77, 104, 121, 143, 169, 195, 210, 224, 225, 256, 289, 320, 323, 246, 410, 512,
           779, 994, 1000, 1021, 1024]


@pytest.mark.parametrize("prec,tol", [(0, 1e-13), (1, 3e-6)])
@pytest.mark.parametrize("n", LENGTHS)
def test_stage_lengths_against_numpy(capi, n, prec, tol):
    for shape in ((n, 3, 6), (2, n, 9), (5, 3, n)):
        x = np.random.default_rng(n).standard_normal(shape)
        k, back = _run(capi, prec, shape, x)
        ref = np.fft.rfftn(x)
        assert np.abs(k - ref).max() <= tol * np.abs(ref).max() * np.log2(x.size + 1), shape
        assert np.abs(back / x.size - x).max() <= tol * np.abs(x).max() * np.log2(x.size + 1), shape
