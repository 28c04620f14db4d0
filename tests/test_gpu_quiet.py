"""Sparse systems above the register loop's size: the particles nothing can touch advanced in flights,
the others step by step (dem_flight.cuh), against the three-kernel step (cooperative_loop 2), bit for
bit: runs around a flight's length, rebuilds, held particles, scenes, and systems that are not quiet."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_idx", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z",
          "tng_sw_x", "tng_sw_y", "tng_sw_z")


def _same(sc, steps, fields=None, **kw):
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, cooperative_loop=coop, **kw)
        for f, v in (fields or {}).items():
            s.particles.set(f, v)
        for k in steps:
            s.run_steps(k)
        out.append((s.particles.download(), s.energy(), s.stats(), s.last_status))
    (a, ea, sa, la), (b, eb, sb, lb) = out
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    assert np.allclose(ea, eb, rtol=1e-12) and la == lb and sa["steps"] == sb["steps"]
    return a, sa, sb


def _lattice(n, vmax=0.5, seed=6):
    sc = S.hcp_box(n=n, seed=seed, vmax=vmax)
    sc.state.omega[:] = np.random.default_rng(seed).uniform(-50, 50, sc.state.omega.shape)
    sc.walls.x[:] += 1.198e-3 * sc.walls.normal    # within micrometres of the largest outer spheres
    return sc


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
def test_flights_equal_single_steps(precision):
    sc = _lattice(60_001)
    a, sa, sb = _same(sc, (1, 2, 63, 64, 65, 130), precision=precision)
    assert sa["cooperative_loop"] == 1 and sa["launches"] < sb["launches"] / 4
    assert a.tng_count.sum() > 0 and np.abs(a.tng_sw_x).max() > 0
    if precision == _lib.DEM_FP64:
        b, _, _ = _same(sc, (130,))
        ref = sc.state.copy()
        O.run(ref, sc.walls, sc.params, sc.dt, 130, skin=sc.skin, gravity=sc.gravity, pow_mode=O.POW_SQRT)
        for f in ("x", "u", "omega", "force", "torque", "tng_count"):
            assert np.array_equal(getattr(b, f), getattr(ref, f)), f


def test_rebuilds_and_held_particles():
    sc = _lattice(70_003, vmax=1.5)
    fix = np.where(np.random.default_rng(2).random(70_003) < 0.2, 1, 0).astype(np.uint8)
    a, sa, sb = _same(sc, (200, 301), fields=dict(fix=fix))
    assert sa["cooperative_loop"] == 1 and sa["rebuilds"] >= 3


def test_oblique_gravity():
    sc = _lattice(60_500)
    sc.gravity = (3.0, 0.0, -9.0)
    _, sa, _ = _same(sc, (150,))
    assert sa["cooperative_loop"] == 1


def test_scenes():
    parts = [_lattice(31_000, seed=k) for k in (1, 2)]
    sc = S.combine_scenes(parts)
    sc.state.omega[:] = 20.0
    _, sa, _ = _same(sc, (140,))
    assert sa["cooperative_loop"] == 1


def test_not_quiet():
    """A squeezed lattice: too many particles close to one another; and an external force."""
    sc = _lattice(60_001)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * 0.93
    _same(sc, (40,))
    n = 66_000
    sc = _lattice(n)
    ext = np.random.default_rng(4).normal(0.0, 1e-3, (n, 3))
    _same(sc, (40,), fields=dict(ext_force=ext))


def test_fast_particles_among_the_others():
    """One held sphere slides along the floor at 50 m/s: the list lasts some twenty steps, quiet classes a
    quarter of that.  They are not worth their builds."""
    n = 60_500
    sc = _lattice(n, vmax=0.05)
    sc.walls.x[4, 2] -= 4e-3                                     # room for it under the lattice
    sc.state.x[0] = sc.state.x[:, :2].min(axis=0).tolist() + [sc.walls.x[4, 2] + sc.state.rad[0] - 1e-6]
    sc.state.u[0] = (50.0, 0.0, 0.0)
    fix = np.zeros(n, np.uint8)
    fix[0] = 3
    _, sa, sb = _same(sc, (300,), fields=dict(fix=fix))
    assert sb["rebuilds"] >= 14 and sa["rebuilds"] == sb["rebuilds"]


def test_speeds_that_rise_after_the_build():
    """A squeezed lattice at rest: the first build finds quiet particles, the release of the contacts ends
    its classes early.  Such a build is one more than without classes, at most one in seventeen."""
    sc = _lattice(60_001, vmax=0.1)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * 0.975
    _, sa, sb = _same(sc, (400,))
    assert sb["rebuilds"] >= 10 and sa["rebuilds"] <= sb["rebuilds"] + 1 + sb["rebuilds"] // 17
