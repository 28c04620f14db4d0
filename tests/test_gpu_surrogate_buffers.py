"""The surrogate's growing device buffers: what one call makes larger or fails to get, the next call
on the same object does not trip over."""
import numpy as np
import pytest
import torch

from cabanadem_b200 import _lib, api, scenarios as S, surrogate as SG

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


@pytest.mark.parametrize("nth", [1, 4, 8, 9, 11, 14])
def test_prediction_after_one_that_ran_out_of_memory(nth):
    """The edges' buffers (eight) and the projection's (six) grow for a larger frame; where one of them
    cannot be had, the call reports it and the object still predicts."""
    ctx = api.Context(0)
    sg = _surrogate(ctx)
    with torch.cuda.stream(sg.stream):
        small, large = _frame(300, "cuda"), _frame(4000, "cuda")

    def predict(s, t):
        return s.predict(t[0], t[1], t[3]).cpu().numpy()

    before = predict(sg, small)
    assert _lib.lib().dem_ctx_debug_fail_alloc(ctx.h, nth) == 0
    with pytest.raises(_lib.DemError, match="out of memory"):
        predict(sg, large)
    assert np.array_equal(predict(sg, small), before)
    fresh = _surrogate(ctx)
    assert np.array_equal(predict(sg, large), predict(fresh, large))
    sg.close()
    fresh.close()
    ctx.close()


@pytest.mark.parametrize("nth", [1, 8, 9, 20, 25])
def test_training_after_a_call_that_ran_out_of_memory(nth):
    ctx = api.Context(0)
    sg = _surrogate(ctx)
    with torch.cuda.stream(sg.stream):
        small, large = _frame(300, "cuda"), _frame(4000, "cuda")
    before = sg.loss_grad(*small)
    assert _lib.lib().dem_ctx_debug_fail_alloc(ctx.h, nth) == 0
    with pytest.raises(_lib.DemError, match="out of memory"):
        sg.loss_grad(*large)
    after = sg.loss_grad(*small)
    assert after[0] == before[0] and np.array_equal(after[1], before[1])
    fresh = _surrogate(ctx)
    got, want = sg.loss_grad(*large), fresh.loss_grad(*large)
    assert got[0] == want[0] and np.array_equal(got[1], want[1])
    sg.close()
    fresh.close()
    ctx.close()
