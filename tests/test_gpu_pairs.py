"""The pair-parallel step's contact search (dem_pairs.cuh) where its first slots, list entries and kept
partners (6, 8 and 8) run out: packings with up to twelve contacts each that come apart again, against
the oracle and the one-kernel step, bit for bit."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FIELDS = ("x", "u", "omega", "force", "torque", "tng_idx", "tng_count", "tng_ss_x", "tng_ss_y", "tng_ss_z",
          "tng_sw_x", "tng_sw_y", "tng_sw_z")
STEPS = (1, 1, 8, 30, 60)


def _packing(n, squeeze):
    sc = S.hcp_box(n=n, seed=11, vmax=2.0)
    c = sc.state.x.mean(axis=0)
    sc.state.x[:] = c + (sc.state.x - c) * squeeze
    sc.state.omega[:] = np.random.default_rng(11).uniform(-50, 50, sc.state.omega.shape)
    sc.walls.x[:] += 1.5e-3 * sc.walls.normal
    return sc


@pytest.mark.parametrize("precision", [_lib.DEM_FP64, _lib.DEM_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,squeeze", [(31, 0.9), (129, 0.9), (2000, 0.9), (2000, 0.95)])
def test_search_equals_the_one_kernel_step(n, squeeze, precision):
    runs = []
    for kw in (dict(dense_form=2), dict(dense_form=1, cooperative_loop=2)):
        sc = _packing(n, squeeze)
        s = api.from_scenario(sc, precision=precision, **kw)
        peak = []
        for k in STEPS:
            s.run_steps(k)
            peak.append(int(s.particles.get("tng_count").max()))
        runs.append((s.particles.download(), s.last_status, s.stats()["rebuilds"]))
    (a, la, ra), (b, lb, rb) = runs
    for f in FIELDS:
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
    assert la == lb and ra == rb
    if n == 2000 and squeeze == 0.9:
        assert max(peak) > 8 and a.tng_count.max() < max(peak)   # more than the kept partners; some ended
    if precision == _lib.DEM_FP64:
        sc = _packing(n, squeeze)
        for k in STEPS:
            O.run(sc.state, sc.walls, sc.params, sc.dt, k, skin=sc.skin, gravity=sc.gravity, pow_mode=O.POW_SQRT)
        for f in ("x", "u", "omega", "force", "torque", "tng_count"):
            assert np.array_equal(getattr(a, f), getattr(sc.state, f)), f
