"""Values that the entry points do not check -- masses that are not finite, positions of gravity_direct that are
not -- come back as results that are not finite; no table is indexed by them, and the next call is unharmed."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_FP64_GROUP, L.PREC_FP32])
def test_masses(precision, value, cuda_lib):
    ic = ics.grid_box(n1=12, seed=5, pmgrid=24)
    with GravityTree(ics.params_for(ic, precision=precision)) as t:
        good = t.compute_grav_accelerations(ic["pos"], ic["mass"], ic["softtype"])
        mass = ic["mass"].copy()
        mass[700] = value
        acc, _, _, _ = t.compute_grav_accelerations(ic["pos"], mass, ic["softtype"])
        d = np.abs(ic["pos"] - ic["pos"][700])
        near = np.linalg.norm(np.minimum(d, 1 - d), axis=1) < 0.5 * ic["rcut"]
        assert not np.isfinite(acc[near]).all(axis=1).any()
        again = t.compute_grav_accelerations(ic["pos"], ic["mass"], ic["softtype"])
    for a, b in zip(good, again):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_positions_of_gravity_direct(value, cuda_lib):
    ic = ics.grid_box(n1=8, seed=6, pmgrid=16)
    with GravityTree(ics.params_for(ic)) as t:
        good = t.gravity_direct(ic["pos"], ic["mass"], ic["softtype"])
        pos = ic["pos"].copy()
        pos[100, 1] = value
        acc, _ = t.gravity_direct(pos, ic["mass"], ic["softtype"])
        others = np.arange(len(pos)) != 100
        assert np.isfinite(acc[100]).all() == False  # noqa: E712
        if value == np.inf:  # an infinitely distant particle pulls nobody
            assert np.isfinite(acc[others]).all()
        else:
            assert np.isnan(acc[others]).any(axis=1).all()
        again = t.gravity_direct(ic["pos"], ic["mass"], ic["softtype"])
    for a, b in zip(good, again):
        assert np.array_equal(a, b)
