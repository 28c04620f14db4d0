"""The step loop that keeps each particle in a thread's registers (dem_live.cuh) against graph
replays of the per-step kernels (cooperative_loop 2), bit for bit: block edges, runs of odd and even
length, lists longer than the marks of a step, external forces, held particles, several materials
and batched scenes."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_idx", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z",
          "tng_sw_x", "tng_sw_y", "tng_sw_z")


def _box(n, seed=5, vmax=2.0, squeeze=0.97):
    sc = S.hcp_box(n=n, seed=seed, vmax=vmax)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * squeeze
    sc.state.omega[:] = np.random.default_rng(seed).uniform(-50, 50, sc.state.omega.shape)
    sc.walls.x[:] += 1.5e-3 * sc.walls.normal
    return sc


def _same(sc, steps, fields=None, **kw):
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, cooperative_loop=coop, **kw)
        for f, v in (fields or {}).items():
            s.particles.set(f, v)
        for k in steps:
            s.run_steps(k)
        out.append((s, s.particles.download(), s.energy(), s.stats(), s.last_status))
    (s, a, ea, sa, la), (_, b, eb, sb, lb) = out
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    assert np.array_equal(ea, eb) and la == lb
    assert sa["cooperative_loop"] == 1 and sb["cooperative_loop"] == 0 and sa["rebuilds"] == sb["rebuilds"]
    return a, sa


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 127, 129, 3001])
def test_loop_equals_graph(n, precision):
    sc = _box(n)
    a, _ = _same(sc, (1, 2, 97, 60), precision=precision)
    if n > 100:
        assert a.tng_count.sum() > 0
    if precision == _lib.DEM_FP64:
        b, _ = _same(sc, (160,))
        ref = sc.state.copy()
        O.run(ref, sc.walls, sc.params, sc.dt, 160, skin=sc.skin, gravity=sc.gravity, pow_mode=O.POW_SQRT)
        for f in ("x", "u", "omega", "force", "torque", "tng_count"):
            assert np.array_equal(getattr(b, f), getattr(ref, f)), f


def test_long_lists():
    sc = _box(900)
    sc.skin = 2.5e-3
    _, st = _same(sc, (80,), max_neighbors=64)
    assert st["max_neighbors"] > 34


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
def test_hooks_and_materials(precision):
    sc = _box(700)
    rng = np.random.default_rng(3)
    soft = rng.random(700) < 0.4
    sc.state.E[soft], sc.state.G[soft] = 1e9, 0.4e9
    fix = np.where(rng.random(700) < 0.1, 3, 0).astype(np.uint8)
    ext = rng.normal(0.0, 2e-3, (700, 3))
    _same(sc, (50, 33), fields=dict(ext_force=ext, fix=fix), precision=precision)


def test_scenes():
    sc = S.batched_scenes(nscenes=7, nmin=70, nmax=400, seed=9)
    sc.state.omega[:] = np.random.default_rng(1).uniform(-50, 50, sc.state.omega.shape)
    a, _ = _same(sc, (300, 301))
    assert a.tng_count.sum() > 0


@pytest.mark.parametrize("quirks", [0x3F, 0x00])
def test_wall_history(quirks):
    """Spheres rolling and bouncing along the floor: wall history kept, cleared and taken up again."""
    sc = _box(400, squeeze=1.0, vmax=0.0)
    sc.params["quirks"] = quirks
    sc.state.x[:, 2] = sc.walls.x[4, 2] + sc.state.rad * (1.0 + 2e-5 * np.arange(400) / 400)
    k = np.arange(400)
    sc.state.x[:, 0], sc.state.x[:, 1] = (k % 20) * 2.6e-3, (k // 20) * 2.6e-3
    sc.walls.x[[0, 2]] = -5e-3
    sc.walls.x[[1, 3]] = 60e-3
    sc.state.u[:, 2], sc.state.u[:, 0] = -0.4, 1.5
    sc.gravity = (0.0, 0.0, -9.81)
    a, _ = _same(sc, (61, 140))
    assert np.abs(a.tng_sw_x).max() > 0


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n", [57_000, 130_001])
def test_several_particles_per_thread(n, precision):
    """More particles than resident threads, few of them in contact, none of them quiet (a thick skin)."""
    sc = S.hcp_box(n=n, seed=3, vmax=2.0)
    sc.skin = 4e-4
    sc.state.omega[:] = np.random.default_rng(3).uniform(-50, 50, sc.state.omega.shape)
    sc.walls.x[:] += 1.198e-3 * sc.walls.normal
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, cooperative_loop=coop, precision=precision)
        for k in (1, 2, 150, 57):
            s.run_steps(k)
        out.append((s.particles.download(), s.stats()))
    (a, sa), (b, sb) = out
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    assert sa["cooperative_loop"] == 1 and sb["cooperative_loop"] == 0 and a.tng_count.sum() > 50


def test_from_sparse_to_dense():
    """A lattice that is squeezed until its steps are too dense for several particles per thread."""
    sc = _box(58_001, squeeze=0.9, vmax=0.5)
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, cooperative_loop=coop)
        s.run_steps(60)
        out.append((s.particles.download(), s.last_status))
    for f in FIELDS:
        assert np.array_equal(getattr(out[0][0], f), getattr(out[1][0], f)), f
    assert out[0][1] == out[1][1] and out[0][0].tng_count.mean() > 1.0
