"""Velocities that become NaN between list builds (a contact with a spin that is one): every form of
the step loop goes on as the per-step kernels do (cooperative_loop 2), until the next build reports
it, and leaves the same state."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z")


def _steps(s, n):
    """The error's name, or None."""
    try:
        s.run_steps(n)
    except _lib.DemError as e:
        return [k for k in _lib.ERR.values() if k in str(e)]
    return None


def _lattice(n, squeeze):
    sc = S.hcp_box(n=n, seed=5, vmax=0.5)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * squeeze
    return sc


@pytest.mark.parametrize("n,squeeze,skin", [(3001, 0.985, None), (60_001, 0.997, None), (130_001, 0.997, 1e-3)],
                         ids=["one_per_thread", "quiet", "several_per_thread"])
def test_contact_loops(n, squeeze, skin):
    sc = _lattice(n, squeeze)
    if skin:
        sc.skin = skin
    s = api.from_scenario(sc, cooperative_loop=2)
    s.run_steps(12)
    hit = int(np.flatnonzero(s.particles.get("tng_count"))[0])   # in contact within the first twelve steps
    sc.state.omega[hit, 1] = np.nan
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, cooperative_loop=coop)
        seen, built = _steps(s, 14), s.stats()["rebuilds"]
        first = s.particles.download()
        out.append((first, seen, built, _steps(s, 600), s.particles.download(), s.stats()))
    (a, ea, ba, fa, la, sa), (b, eb, bb, fb, lb, sb) = out
    assert ea is None and eb is None and ba == bb == 1
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f), equal_nan=True), f
    assert np.isnan(a.x[hit]).all() and np.isfinite(a.x).mean() > 0.99
    assert fa == fb and sa["steps"] == sb["steps"]
    assert fa == ["DEM_ERR_NAN"] or skin   # the thick skin lasts
    assert sa["cooperative_loop"] == 1 and sb["cooperative_loop"] == 0


def test_rebuild_every_step():
    sc = _lattice(900, 0.97)
    sc.delta = 3.6e-3
    sc.state.u[17, 1] = np.nan
    out = []
    for coop in (0, 2):
        s = api.from_scenario(sc, rebuild_every_step=True, cooperative_loop=coop)
        out.append((_steps(s, 30), s.particles.download(), s.stats()["steps"]))
    (ea, a, na), (eb, b, nb) = out
    assert ea == eb and na == nb
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f), equal_nan=True), f


def test_bonded_loops():
    case = S.bonded_bar(nx=20, ny=6, nz=4)
    case["state"].u[100, 0] = np.nan
    got = []
    for chunk in (0, 8):
        bonds = api.bonded_from_case(case, steps_per_launch=chunk)
        bonds.run_steps(3)
        p = bonds.solver.particles
        got.append([p.get(f) for f in ("x", "u", "omega", "force", "torque")] + [bonds.solver.stats()["steps"]])
    for a, b in zip(*got):
        assert np.array_equal(a, b, equal_nan=True)
    assert 0 < np.isnan(got[0][0]).sum() < got[0][0].size
