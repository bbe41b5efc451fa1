"""The tile autotuner times the fixed rule's own tile among its candidates,
also where it is no power of two, so that its choice is never slower."""
import math
import re

import pytest

from conftest import params_for
from test_gpu_parity import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n", [(0, 44), (1, 52)])
def test_rule_is_a_candidate(capi, prec, n):
    from cuda_sto_pf_gb300.solver import Solver
    p = params_for(capi, "c2.params", n=n, precision=prec, fft_autotune=3, elastic_fail_on_nonconvergence=0)
    phi, xB, _ = _inputs(capi, p, n, False, seed=31)
    with Solver(p) as s:
        s.load(phi, xB)
        s.step(1)
    rows = re.findall(r"^\S+ n=%d \S+ tile=(\d+) (\S+) ms rule=(\d+) (\S+) ms$" % n, capi.tile_report(), re.M)
    assert len(rows) >= 4
    assert any(int(rule) & (int(rule) - 1) for _, _, rule, _ in rows)   # one that is no power of two
    for tile, t, rule, t_rule in rows:
        assert math.isfinite(float(t_rule)) and float(t) <= float(t_rule), (tile, t, rule, t_rule)
