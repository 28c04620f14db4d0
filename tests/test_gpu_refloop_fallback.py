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


def test_full_cells_are_not_tried_in_every_run():
    """Some 20 spheres in a cell: the loop takes no step, and runs of one step go straight to the graph
    after one that found that out."""
    sc = _box(900, 6e-3)
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, rebuild_every_step=True, cooperative_loop=coop, max_neighbors=128)
        s.run_steps(1)
        before = s.stats()["launches"]
        for _ in range(33):
            s.run_steps(1)
        assert s.stats()["cooperative_loop"] == 0
        out.append((s.stats()["launches"] - before, _state(s)))
    (la, a), (lb, b) = out
    assert lb < la <= lb + 2 * 6   # an attempt is six launches; one in every 17 runs
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_a_cell_that_fills_up_in_the_middle_of_a_run():
    """Spheres with a thin cutoff that fly together: the loop takes the first steps, a cell becomes full,
    the loop starts again on a fresh grid and the graph takes what it cannot do."""
    n, r = 216, 1e-3
    sc = S.hcp_box(n=n, seed=4, vmax=0.0)
    k = np.arange(n)
    sc.state.rad[:] = 0.05 * r                         # small spheres ...
    sc.state.rad[0] = r                                # ... and a large one, which makes the cells wide
    sc.state.x[:] = np.stack([k % 6, (k // 6) % 6, k // 36], axis=1) * 2.0 * r + 3e-3
    sc.state.x[0] = sc.state.x.max(axis=0) + 8e-3
    sc.state.u[:] = -(sc.state.x - sc.state.x[1:].mean(axis=0)) * 2000.0
    sc.state.u[0] = 0.0
    sc.walls.x[:] -= 1.0 * sc.walls.normal
    sc.delta, sc.gravity = 3e-3, (0.0, 0.0, 0.0)
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, rebuild_every_step=True, cooperative_loop=coop, max_neighbors=128)
        s.run_steps(4000)
        out.append((_state(s), s.stats()))
    (a, sa), (b, sb) = out
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert sa["cooperative_loop"] == 1 and sb["cooperative_loop"] == 0
    # both forms took steps: more launches than the loop alone, far fewer than the graph (14 per step)
    assert 4000 < sa["launches"] < sb["launches"] - 14 * 1000
