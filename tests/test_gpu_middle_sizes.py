"""Systems a little larger than the particles resident at once (56,832), from sparse to dense: the forms
that the step goes through are chosen by what is in contact and how long the lists are, with the same
results as the per-step kernels, and a dense step is not one kernel that one more block makes wait."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_idx", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z",
          "tng_sw_x", "tng_sw_y", "tng_sw_z")


def _box(n, squeeze, skin=None):
    sc = S.hcp_box(n=n, seed=7, vmax=0.3)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * squeeze
    sc.state.omega[:] = np.random.default_rng(7).uniform(-50, 50, sc.state.omega.shape)
    sc.walls.x[:] += 1.2e-3 * sc.walls.normal
    if skin:
        sc.skin = skin
    return sc


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,squeeze,skin", [(56_832, 0.92, None), (56_833, 0.92, None), (65_537, 0.95, 4e-4),
                                            (150_001, 0.98, 4e-4), (200_003, 0.98, 2e-4)])
def test_forms_agree(n, squeeze, skin, precision):
    sc = _box(n, squeeze, skin)
    runs = []
    for kw in (dict(), dict(cooperative_loop=2), dict(dense_form=1, cooperative_loop=2)):
        s = api.from_scenario(sc, precision=precision, **kw)
        for k in (1, 40, 25):
            s.run_steps(k)
        runs.append((s.particles.download(), s.last_status, s.stats()))
        s.close()
    a, la, sa = runs[0]
    assert a.tng_count.mean() > 0.02
    for b, lb, _ in runs[1:]:
        assert la == lb
        for f in FIELDS:
            assert np.array_equal(getattr(a, f), getattr(b, f)), f


def test_a_dense_step_above_the_resident_size_is_three_kernels():
    launches = {}
    for coop in (0, 2):
        s = api.from_scenario(_box(56_900, 0.92), cooperative_loop=coop)
        s.run_steps(30)                      # the density is known after some steps
        a = s.stats()
        s.run_steps(30)
        b = s.stats()
        assert b["cooperative_loop"] == 0
        # without the builds (20 kernels each), the run's two and the loop's control kernels
        launches[coop] = (b["launches"] - a["launches"] - 20 * (b["rebuilds"] - a["rebuilds"])) / 30
        s.close()
    assert 3.0 <= launches[0] < 4.5 and launches[2] < 2.5   # graphs alone stay with one kernel


@pytest.mark.parametrize("skin,loop", [(1e-4, 1), (2e-4, 0)], ids=["thin", "thick"])
def test_long_lists_leave_the_loop_with_fewer_contacts(skin, loop):
    """Four particles per thread, between a 32nd and a 16th of them in contact: the several-per-thread loop
    with less than one listed partner each, the three-kernel step with two."""
    sc = _box(200_003, 0.98, skin)
    sc.state.u[:] = 0.0
    s = api.from_scenario(sc)
    s.run_steps(1)
    assert s.stats()["cooperative_loop"] == 1   # from here on, or not
    s.run_steps(29)
    s.run_steps(10)
    share = (s.particles.get("tng_count") > 0).mean()
    assert 1 / 32 < share < 1 / 16
    assert s.stats()["cooperative_loop"] == loop
