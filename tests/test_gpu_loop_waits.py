"""The bounded waits of the resident step loops and of the staged bonded step: with
dem_solver_debug_stream_waits(drop_copies=1) no block arrives at its barrier and no copy is issued, so
every wait gives up after the poll limit with nothing in flight, and the run ends with DEM_ERR_TIMEOUT.
With the default bounds back and the state set again the same object steps as the per-step kernels do."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_idx", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z")
HIST = ("ft_x", "ft_y", "ft_z", "mn_x", "mn_y", "mn_z", "mt_x", "mt_y", "mt_z")


def _timed_out(h, run):
    L = _lib.lib()
    assert L.dem_solver_debug_stream_waits(h, 64, 1) == 0
    try:
        with pytest.raises(_lib.DemError, match="DEM_ERR_TIMEOUT"):
            run()
    finally:
        assert L.dem_solver_debug_stream_waits(h, 0, 0) == 0


@pytest.mark.parametrize("n,skin,kw", [(3001, None, {}), (60_001, None, {}), (130_001, 1e-3, {}),
                                       (3001, None, dict(rebuild_every_step=True))],
                         ids=["one_per_thread", "quiet", "several_per_thread", "rebuild_every_step"])
def test_contact_loops(n, skin, kw):
    sc = S.hcp_box(n=n, seed=5, vmax=0.5)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * (0.97 if n == 3001 else 0.997)
    if skin:
        sc.skin = skin
    if kw:
        sc.delta = 3.6e-3
    s = api.from_scenario(sc, **kw)
    s.run_steps(20)
    assert s.stats()["cooperative_loop"] == 1
    _timed_out(s.h, lambda: s.run_steps(5))
    s.particles.upload(sc.state)
    s.run_steps(40)
    assert s.stats()["cooperative_loop"] == 1
    b = api.from_scenario(sc, cooperative_loop=2, **kw)
    b.run_steps(40)
    x, y = s.particles.download(), b.particles.download()
    for f in FIELDS:
        assert np.array_equal(getattr(x, f), getattr(y, f)), f


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("chunk,max_bonds", [(0, 6), (8, 6), (8, 3)], ids=["loop", "tiles", "tiles_in_one_ring"])
def test_bonded_forms(chunk, max_bonds, precision):
    case = S.bonded_bar(nx=20, ny=6, nz=4) if max_bonds == 6 else S.bonded_bar(nx=300, ny=1, nz=1)
    bonds = api.bonded_from_case(case, steps_per_launch=chunk, precision=precision)
    p, start = bonds.solver.particles, {k: bonds.get(k) for k in HIST + ("broken",)}
    bonds.run_steps(20)
    _timed_out(bonds.solver.h, lambda: bonds.run_steps(5))
    for f in ("x", "u", "omega", "force", "torque"):
        p.set(f, getattr(case["state"], f))
    for k, v in start.items():
        bonds.set(k, v)
    bonds.run_steps(30)
    fresh = api.bonded_from_case(case, steps_per_launch=chunk, precision=precision)
    fresh.run_steps(30)
    for f in ("x", "u", "omega", "force", "torque"):
        assert np.array_equal(p.get(f), fresh.solver.particles.get(f)), f
    for k in start:
        assert np.array_equal(bonds.get(k), fresh.get(k)), k
