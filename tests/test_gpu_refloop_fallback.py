"""The rebuild-every-step loop (dem_refloop.cuh) where it cannot go on: tables that cannot be had, cells
that fill up in the middle of a run or in every step.  The graph of build and step kernels
(cooperative_loop 2) takes the steps left, with the same results."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_idx", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z")


def _box(n, delta, vmax=0.5):
    sc = S.hcp_box(n=n, seed=5, vmax=vmax)
    sc.delta = delta
    return sc


def _state(s):
    a = s.particles.download()
    return [getattr(a, f) for f in FIELDS] + [np.array(s.stats()["steps"])]


@pytest.mark.parametrize("nth", [1, 2, 3])
def test_no_memory_for_the_tables(nth):
    sc = _box(700, 3.6e-3)
    ctx = api.Context(0)
    s = api.from_scenario(sc, ctx=ctx, rebuild_every_step=True)
    assert _lib.lib().dem_ctx_debug_fail_alloc(ctx.h, nth) == 0
    s.run_steps(10)
    assert s.stats()["cooperative_loop"] == 0
    s.run_steps(7)
    b = api.from_scenario(sc, rebuild_every_step=True, cooperative_loop=2)
    b.run_steps(10)
    b.run_steps(7)
    for x, y in zip(_state(s), _state(b)):
        assert np.array_equal(x, y)
    s.close()
    ctx.close()
