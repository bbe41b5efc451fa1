"""Gradient clipping over the range of float gradients: entries whose squares
overflow a float are clipped as any others."""
import numpy as np
import pytest

from test_fno import _cfg, _dev, _model, _weights, fo

pytestmark = pytest.mark.gpu


# a target's size sets the gradient's: the loss is relative to the target's
# square.  Tolerance as for the unclipped step (test_fno.py): the clip factor
# and the scaled gradient each add one rounding to float.
@pytest.mark.parametrize("target,large", [(1.0, False), (2.5e-12, True)])
def test_clipped_step_matches_reference(capi, target, large):
    rng = np.random.default_rng(41)
    cfg = _cfg((8, 8, 8), 2, 1, rng)
    w = _weights(cfg, rng)
    a, t = rng.normal(size=(8, 8, 8, 8)), target * rng.normal(size=(3, 8, 8, 8))
    lr, b1, b2, eps, wd = 1e-2, 0.9, 0.99, 1e-8, 1e-3
    with _model(capi, cfg, w) as m:
        m.loss_grad(_dev(a), _dev(t))
        g = m.grad().astype(np.float64)
        norm = np.linalg.norm(g)
        assert np.isfinite(norm) and (np.abs(g).max() > 2e19) == large
        clip = float(np.float32(0.25 * norm)) if not large else 1.0
        m.adam_step(lr, b1, b2, eps, wd, clip_norm=clip)
        want, _, _ = fo.adam_reference(w.astype(np.float64), g * (clip / norm), np.zeros(w.size), np.zeros(w.size), 1,
                                       lr, b1, b2, eps, wd)
        assert np.abs(m.params() - want).max() <= 2e-6 * max(1.0, np.abs(want).max())
