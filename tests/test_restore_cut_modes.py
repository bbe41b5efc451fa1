"""A restored displacement holds the modes of the 2/3 rule only: content that a
checkpoint carries outside them is dropped, and the run goes on as without it."""
import ctypes

import numpy as np
import pytest

from conftest import params_for
from test_checkpoint import _State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 21])
def test_restore_drops_cut_modes(capi, tmp_path, n):
    from cuda_sto_pf_gb300 import workloads
    from cuda_sto_pf_gb300.solver import Solver
    lib = capi.load()
    shape = (n, n, n)
    st = _State(capi, shape)
    p = st.p
    p.zero_mode_enabled = 1
    capi.finalize(p)
    rng = np.random.default_rng(5)
    w = workloads.single_sphere(n=n, radius=4.0)
    phi, xB = w["phi"], w["xB"]
    lib.pfgb_prepare_raw_fields(ctypes.byref(p), 0.07, phi.ctypes.data, xB.ctypes.data, None, None, phi.size)
    path, other = str(tmp_path / "a.ckpt"), str(tmp_path / "b.ckpt")
    with Solver(p) as s:
        s.load(phi, xB)
        s.step(2)
        s.checkpoint_save(path, initial_state_class="RANDOM")
    out = st.empty(capi)
    capi.check(lib.pfgb_checkpoint_provenance_for(ctypes.byref(p), b"RANDOM", None, None,
                                                  ctypes.byref(out.provenance)), "provenance_for")
    prov = out.provenance
    capi.check(lib.pfgb_checkpoint_read_file(path.encode(), ctypes.byref(prov), ctypes.byref(out)), "read")
    nx, ny, nz = shape
    nzc = nz // 2 + 1
    wave = lambda n: np.minimum(np.arange(n), n - np.arange(n)) * 3 >= n
    cut = np.zeros((nx, ny, nzc), bool)
    cut[:, wave(ny)] = True
    cut[..., np.arange(nzc) * 3 >= nz] = True
    u = st.ou.reshape(3, nx, ny, nzc, 2)
    assert not u[:, cut].any()
    u[:, cut] = rng.standard_normal((3, int(cut.sum()), 2))
    capi.check(lib.pfgb_checkpoint_write_file(other.encode(), ctypes.byref(out)), "write")
    res = []
    for f in (path, other):
        with Solver(p) as s:
            s.checkpoint_restore(f, initial_state_class="RANDOM")
            s.step(1)
            res.append((s.fields(), s.displacement_k()))
    for k in ("phi", "xB", "Y"):
        assert np.array_equal(res[0][0][k], res[1][0][k]), k
    assert np.array_equal(res[0][1], res[1][1])
