"""The learned start's kernels at the edges of their tiles, against the float64
oracle: an odd z axis (cells taken one by one, not in pairs), a last tile of
cells that is partly empty, a z axis one position past a staged chunk, an odd
number of modes, a y axis of two chunks of twiddles.  Tolerances as on the
regular shapes (test_fno.py): FP32 sums forward, central differences for
gradients."""
import numpy as np
import pytest

from conftest import rel_l2
from test_fno import _cfg, _dev, _model, _weights, fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,modes,layers", [((5, 6, 9), 2, 2), ((4, 3, 65), 1, 1), ((10, 11, 64), 5, 2),
                                                ((2, 2, 2), 1, 1), ((2, 520, 3), 1, 1)], ids=str)
def test_forward_and_gradients_at_tile_edges(capi, shape, modes, layers):
    import torch
    rng = np.random.default_rng(31)
    cfg = _cfg(shape, modes, layers, rng)
    w = _weights(cfg, rng)
    wr = fo.round_weights(w, cfg)
    a, t = rng.normal(size=(8,) + shape), rng.normal(size=(3,) + shape)
    with _model(capi, cfg, w) as m:
        out = torch.empty((3,) + shape, device="cuda")
        m.forward(_dev(a), out)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        loss = m.loss_grad(_dev(a), _dev(t))
        g = m.grad()
    assert rel_l2(got, fo.forward(wr, a, cfg)) <= 2e-6
    want = fo.loss(wr, a, t, cfg)
    assert abs(loss - want) <= 1e-5 * want
    off = fo.offsets(cfg)
    for name, shp, _ in fo.layout(cfg):
        n = int(np.prod(shp))
        idx = off[name] + rng.choice(n, size=min(3, n), replace=False)
        fd = fo.fd_gradient(wr, a, t, cfg, idx, h=1e-4)
        assert np.abs(g[idx] - fd).max() <= 2e-3 * max(np.abs(fd).max(), 1e-6), name
