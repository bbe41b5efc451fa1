"""The learned start's y passes and layer kernel on both sides of the sizes where
their forms change (few_slabs_fwd, few_slabs_inv, few_cells in fno.cu), against the
float64 oracle at the forward test's tolerance."""
import numpy as np
import pytest

from conftest import rel_l2
from test_fno import _cfg, _dev, _model, _weights, fo

pytestmark = pytest.mark.gpu


# 63 | 64 x positions at 12 modes: both y passes' threads fall short of | reach
# 152 x 480; a y axis of 170 | 171 positions there: all twiddles fit | do not; 136 | 137
# positions at 64 x 2 modes: the inverse's threads alone; 38,912 cells: the last
# grid of one cell a thread, then two with an even and an odd z axis; few lines of a long z axis
@pytest.mark.parametrize("shape,modes", [((63, 24, 24), 12), ((64, 24, 24), 12), ((64, 170, 24), 12),
                                         ((64, 171, 24), 12), ((64, 136, 4), 2), ((64, 137, 4), 2), ((152, 16, 16), 2),
                                         ((64, 24, 26), 12), ((65, 24, 25), 12), ((3, 24, 1000), 1)], ids=str)
def test_forward_on_both_sides(capi, shape, modes):
    import torch
    rng = np.random.default_rng(51)
    cfg = _cfg(shape, modes, 2, rng)
    w = _weights(cfg, rng)
    a = rng.normal(size=(8,) + shape)
    with _model(capi, cfg, w) as m:
        out = torch.empty((3,) + shape, device="cuda")
        m.forward(_dev(a), out)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
    assert rel_l2(got, fo.forward(fo.round_weights(w, cfg), a, cfg)) <= 2e-6


@pytest.mark.parametrize("shape", [(152, 16, 16), (64, 24, 26), (65, 24, 25)], ids=str)
def test_gradients_of_every_layer_form(capi, shape):
    """What the layer kernel keeps for the backward pass, in each form; tolerance of
    the central differences as in test_fno.py."""
    rng = np.random.default_rng(52)
    cfg = _cfg(shape, 2, 2, rng)
    w = _weights(cfg, rng)
    wr = fo.round_weights(w, cfg)
    a, t = rng.normal(size=(8,) + shape), rng.normal(size=(3,) + shape)
    with _model(capi, cfg, w) as m:
        loss = m.loss_grad(_dev(a), _dev(t))
        g = m.grad()
    want = fo.loss(wr, a, t, cfg)
    assert abs(loss - want) <= 1e-5 * want
    off = fo.offsets(cfg)
    for name, shp, _ in fo.layout(cfg):
        idx = off[name] + rng.choice(int(np.prod(shp)), size=1)
        fd = fo.fd_gradient(wr, a, t, cfg, idx, h=1e-4)
        assert np.abs(g[idx] - fd).max() <= 2e-3 * max(np.abs(fd).max(), 1e-6), name
