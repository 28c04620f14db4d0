"""The bonded run's forms against the CPU oracle, bit for bit: the register loop (eight lanes per
particle), the staged step (a tile's bonds in shared memory; steps_per_launch set) and, for more than
the ring's slots, tiles with rows left over, around the edges of their blocks and with bonds that break."""
import numpy as np
import pytest

from cabanadem_b200 import _lib, api, scenarios as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu
HIST = ("ft_x", "ft_y", "ft_z", "mn_x", "mn_y", "mn_z", "mt_x", "mt_y", "mt_z")


def _bar(nx, ny, nz, pull=0.05, seed=1, **kw):
    case = S.bonded_bar(nx=nx, ny=ny, nz=nz, pull=pull, **kw)
    rng = np.random.default_rng(seed)
    st = case["state"]
    st.x[:] += rng.uniform(-5e-6, 5e-6, st.x.shape)
    st.u[:] += rng.uniform(-0.01, 0.01, st.u.shape)
    st.omega[:] = rng.uniform(-5, 5, st.omega.shape)
    st.rad[:] *= rng.uniform(0.98, 1.0, st.n)
    return case


def _oracle(case, n):
    st, b = case["state"].copy(), case["bonds"].copy()
    O.setup_bonds(b, st, case["bond_factor"], case["search_cutoff"])
    O.bonded_run(st, b, case["bparams"], case["dt"], n, ext_force=case["ext_force"], fix_flags=case["fix_flags"],
                 pow_mode=O.POW_SQRT)
    return st, b


def _equal(bonds, st, b):
    for f in ("x", "u", "omega", "force", "torque"):
        assert np.array_equal(bonds.solver.particles.get(f), getattr(st, f)), f
    assert np.array_equal(bonds.get("broken"), b.broken)
    for k in HIST:
        assert np.array_equal(bonds.get(k), b.hist[k]), k


@pytest.mark.parametrize("chunk", [0, 16], ids=["loop", "tiles"])
@pytest.mark.parametrize("size", [(2, 1, 1), (17, 1, 1), (5, 5, 5), (8, 4, 4), (43, 3, 1), (13, 5, 3)])
def test_forms_equal_oracle(size, chunk):
    case = _bar(*size)
    st, b = _oracle(case, 60)
    bonds = api.bonded_from_case(case, steps_per_launch=chunk)
    bonds.run_steps(60)
    _equal(bonds, st, b)


@pytest.mark.parametrize("chunk", [0, 32], ids=["loop", "tiles"])
def test_breakage(chunk):
    case = _bar(20, 6, 4, pull=6.0)
    st, b = _oracle(case, 900)
    assert 0 < b.broken.sum() < b.count.sum()
    bonds = api.bonded_from_case(case, steps_per_launch=chunk)
    bonds.run_steps(900)
    _equal(bonds, st, b)


def test_many_bonds_and_forces():
    """Face and edge neighbours bonded: up to 18 bonds, more than the loop's lanes and the ring's slots;
    external forces."""
    case = _bar(9, 7, 5, max_bonds=20)
    case["bond_factor"], case["search_cutoff"] = 3.0, 1.6e-3
    case["ext_force"] = np.random.default_rng(2).normal(0.0, 0.5, (case["state"].n, 3))
    st, b = _oracle(case, 40)
    assert b.count.max() > 12
    bonds = api.bonded_from_case(case)
    bonds.run_steps(40)
    _equal(bonds, st, b)


def test_forms_agree_in_mixed_precision_and_over_several_runs():
    case = _bar(21, 7, 5)
    got = []
    for chunk in (0, 8):
        bonds = api.bonded_from_case(case, precision=_lib.DEM_MIXED, steps_per_launch=chunk)
        for n in (1, 2, 33):
            bonds.run_steps(n)
        got.append([bonds.solver.particles.get(f) for f in ("x", "u", "omega", "force", "torque")] +
                   [bonds.get(k) for k in HIST])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
