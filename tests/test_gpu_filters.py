"""The semi-implicit filters of FP32 runs, num / (1 + m k^2) rounded like the
double quotient, where they damp nothing, a little and all but the mean,
against the oracle at the step parity's tolerance for FP32."""
import numpy as np
import pytest

from conftest import params_for, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kappa", [1e-9, 1.0, 1e7])
def test_fp32_filters_over_their_range(capi, oracle, kappa):
    from cuda_sto_pf_gb300.solver import Solver
    p = params_for(capi, "c2.params", precision=1, model_mode=1, elastic_fail_on_nonconvergence=0)
    p.Nx, p.Ny, p.Nz = 9, 12, 10
    p.kappa_phi = kappa
    capi.finalize(p)
    rng = np.random.default_rng(23)
    phi = rng.uniform(0.1, 0.9, (9, 12, 10))
    xB = rng.uniform(0.02, 0.04, phi.shape)
    eta = rng.uniform(0.0, 0.2, phi.shape)
    o = oracle(p, threads=2)
    o.load(phi, xB, eta)
    assert o.step(1) == 0
    with Solver(p) as s:
        s.load(phi, xB, eta)
        s.step(1)
        f = s.fields()
    fo = o.fields()
    for k in ("phi", "xB", "eta"):
        assert rel_l2(f[k], fo[k]) <= 1e-5, k
