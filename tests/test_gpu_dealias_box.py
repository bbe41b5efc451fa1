"""The passes move only the modes that the 2/3 rule keeps (Grid3): grids whose
box has an edge in every place it can have one, against the oracle, at the
step parity's tolerances."""
import numpy as np
import pytest

from conftest import params_for, rel_l2

pytestmark = pytest.mark.gpu

# axes of length 1 and 2 (one kept mode), 3 (the cut starts at the last mode),
# odd and even ones, a z axis whose kept columns end inside, at and past a
# tile of columns, and the 246-point engine on one axis at a time, its last tile
# of columns full, with a pair and with an odd column left over
SHAPES = [(4, 1, 2), (1, 3, 6), (3, 2, 5), (7, 9, 8), (12, 10, 47), (9, 12, 48), (5, 6, 49), (246, 4, 6), (4, 246, 9),
          (3, 4, 246), (246, 5, 126), (4, 246, 130), (246, 3, 134)]


@pytest.mark.parametrize("prec,tol", [(0, 1e-6), (1, 1e-5)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_step_on_kept_modes(capi, oracle, shape, prec, tol):
    from cuda_sto_pf_gb300.solver import Solver
    p = params_for(capi, "c2.params", precision=prec, model_mode=1, elastic_fail_on_nonconvergence=0)
    p.Nx, p.Ny, p.Nz = shape
    capi.finalize(p)
    rng = np.random.default_rng(17)
    phi = rng.uniform(0.1, 0.9, shape)
    xB = rng.uniform(0.02, 0.04, shape)
    eta = rng.uniform(0.0, 0.2, shape)
    o = oracle(p, threads=2)
    o.load(phi, xB, eta)
    assert o.step(2) == 0
    with Solver(p) as s:
        s.load(phi, xB, eta)
        s.step(2)
        f, u = s.fields(), s.displacement_k()
    fo = o.fields()
    for k in ("phi", "xB", "eta"):
        assert rel_l2(f[k], fo[k]) <= tol, k
    # the displacement outside the box stays zero
    nx, ny, nz = shape
    u = u.reshape(3, nx, ny, nz // 2 + 1)
    wave = lambda n, m: np.minimum(np.arange(m), n - np.arange(m)) * 3 >= n
    assert not u[:, :, wave(ny, ny)].any() and not u[..., np.arange(nz // 2 + 1) * 3 >= nz].any()
