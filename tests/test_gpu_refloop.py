"""The rebuild-every-step mode in one cooperative launch (dem_refloop.cuh) against the graph of
build and step kernels (cooperative_loop 2), bit for bit: sizes around the group shapes' edges,
lists that grow, cells that overflow, particles that leave the launch's grid."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_idx", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z",
          "tng_sw_x", "tng_sw_y", "tng_sw_z")


def _box(n, squeeze=0.97, seed=5, vmax=2.0):
    sc = S.hcp_box(n=n, seed=seed, vmax=vmax)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * squeeze
    sc.state.omega[:] = np.random.default_rng(seed).uniform(-50, 50, sc.state.omega.shape)
    sc.walls.x[:] += 1.5e-3 * sc.walls.normal      # the walls reach the outer spheres
    return sc


def _pair(sc, steps, grown=0, **kw):
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, rebuild_every_step=True, cooperative_loop=coop, **kw)
        for k in steps:
            s.run_steps(k)
        out.append((s, s.particles.download(), s.neighbors(), s.energy(), s.stats()))
    (s, a, na, ea, sa), (_, b, nb, eb, sb) = out
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    assert np.array_equal(na[0], nb[0]) and np.array_equal(na[1], nb[1]) and np.array_equal(ea, eb)
    for k in ("steps", "max_neighbors", "neighbor_capacity", "status"):
        assert sa[k] == sb[k], k
    # the graph counts a build again after each growth of the lists
    assert sa["rebuilds"] == sb["rebuilds"] if grown == 0 else sa["rebuilds"] <= sb["rebuilds"]
    assert sb["cooperative_loop"] == 0
    return s, a, sa


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 7, 33, 1184, 1185, 3552, 3553, 5001])
def test_loop_equals_graph(n, precision):
    sc = _box(n)
    sc.delta = 3.6e-3
    s, a, st = _pair(sc, (1, 3, 36), precision=precision)
    assert st["cooperative_loop"] == 1 and st["rebuilds"] == 40
    if n > 100:
        assert a.tng_count.sum() > 0
    if 100 < n <= 1185:   # the squeezed box of 5,001 has no sphere at a wall
        assert np.abs(a.tng_sw_x).max() > 0
    if precision == _lib.DEM_FP64 and n <= 1185:
        ref = _box(n).state
        O.run(ref, sc.walls, sc.params, sc.dt, 40, delta=sc.delta, gravity=sc.gravity, pow_mode=O.POW_SQRT)
        # the runs are continued: forces of the last step of the first run start the second
        assert np.abs(a.x - ref.x).max() < 1e-12


def test_lists_grow():
    sc = _box(700)
    sc.delta = 4.5e-3
    _, _, st = _pair(sc, (5, 20), grown=1, max_neighbors=4)
    assert st["max_neighbors"] > 8 and st["cooperative_loop"] == 1


def test_full_cell_goes_on_with_the_graph():
    """Spheres much smaller than the cutoff: more than a cell holds."""
    sc = _box(900, squeeze=1.0)
    sc.delta = 6e-3   # some 90 neighbours, 20 spheres in a cell
    _, _, st = _pair(sc, (4, 8), max_neighbors=128)
    assert st["status"] == 0


def test_leaving_the_grid():
    """Two groups flying apart: the grid of the launch is left far behind."""
    sc = _box(200, vmax=0.5)
    sc.delta = 3.6e-3
    sc.walls.x[:] -= 10.0 * sc.walls.normal
    sc.state.u[:100, 0] -= 900.0
    sc.state.u[100:, 0] += 900.0
    _, a, st = _pair(sc, (400,))
    assert np.ptp(a.x[:, 0]) > 0.03 and st["cooperative_loop"] == 1
