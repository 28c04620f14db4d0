"""The surrogate's growing device buffers: what one call makes larger or fails to get, the next call
on the same object does not trip over."""
import numpy as np
import pytest
import torch

from cabanadem_b200 import api, scenarios as S, surrogate as SG

pytestmark = pytest.mark.gpu


def _frame(n, dev, seed=3):
    """Positions at three strides of n disks in a column (one stride apart by a few micrometres)."""
    sc = S.dam_break(n=n, aspect=1.0, seed=seed)
    rng = np.random.default_rng(seed)
    x, d = sc.state.x, rng.normal(0.0, 2e-6, (3, n, 3))
    t = [torch.from_numpy(np.ascontiguousarray(x + d[k])).to(dev) for k in range(3)]
    return t + [torch.from_numpy(sc.state.rad.copy()).to(dev)]


def _surrogate(ctx):
    prm = SG.params_for(S.dam_break(n=64, aspect=1.0), sigma_a=2.0e-4, max_nodes=4096)
    sg = SG.Surrogate(ctx, prm)
    sg.init_params(7)
    return sg


def test_training_buffers_follow_a_prediction_on_more_edges():
    """Training on a few nodes, a prediction on many, training on as many: the last needs larger training
    buffers than the first, though the prediction has already grown the edges'."""
    ctx = api.Context(0)
    sg = _surrogate(ctx)
    with torch.cuda.stream(sg.stream):
        small, large = _frame(300, "cuda"), _frame(4000, "cuda")
    sg.loss_grad(*small)
    sg.predict(large[0], large[1], large[3])
    loss, grad = sg.loss_grad(*large)
    fresh = _surrogate(ctx)
    want = fresh.loss_grad(*large)
    assert loss == want[0] and np.array_equal(grad, want[1])
    sg.close()
    fresh.close()
    ctx.close()
