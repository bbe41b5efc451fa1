"""Standalone transforms from more threads at once than there is kept room for
their tables, each on its own stream, against numpy at the transform tests'
tolerances."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 13])
def test_transforms_from_threads(capi, threads):
    import torch
    lib = capi.load()
    errors = []

    def work(i):
        try:
            rng = np.random.default_rng(i)
            shape = (8 + i, 9 + 2 * i, 10 + 3 * i)
            prec, tol, rt, ct = ((capi.PREC_FP64, 1e-13, torch.float64, torch.complex128),
                                 (capi.PREC_FP32, 3e-6, torch.float32, torch.complex64))[i % 2]
            x = rng.normal(size=shape)
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                d = torch.from_numpy(x).to("cuda", rt)
                want = np.fft.rfftn(d.cpu().numpy().astype(np.float64))
                for _ in range(6):
                    out = torch.empty(want.shape, dtype=ct, device="cuda")
                    back = torch.empty(shape, dtype=rt, device="cuda")
                    capi.check(lib.pfgb_fft3d_r2c(prec, *shape, d.data_ptr(), out.data_ptr(), s.cuda_stream), "r2c")
                    got = out.cpu().numpy()
                    capi.check(lib.pfgb_fft3d_c2r(prec, *shape, out.data_ptr(), back.data_ptr(), s.cuda_stream), "c2r")
                    r = back.cpu().numpy() / x.size
                    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
                    assert np.linalg.norm(r - d.cpu().numpy()) <= tol * np.linalg.norm(x)
        except Exception as e:   # noqa: BLE001 - handed to the test's thread
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[:3]
