"""The PM readout of few particles on a large mesh goes component by component, of more through records of force and
potential.  A massless particle at the end takes a set over the line without changing the mesh; the others'
results agree to the rounding of FP64 sums."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["even", "clustered"])
def test_components_against_records(kind, cuda_lib):
    grid = 400
    n = grid**3 // 128  # the first size with records
    rng = np.random.default_rng(9)
    pos = rng.uniform(0, 1, (n, 3))
    if kind == "clustered":
        pos[: n // 2] = (pos[: n // 2] - 0.5) * 0.01 + 0.999
    pos[:8] = [[i >> 2, i >> 1 & 1, i & 1] for i in range(8)]  # box corners
    mass = rng.uniform(0.5, 1.5, n) / n
    mass[-1] = 0.0
    asmth = 1.25 / grid
    with GravityTree(L.make_params(periodic=True, box_size=1.0, asmth=asmth, rcut=4.5 * asmth, softening=(1e-3,))) as t:
        a, p = t.pm_periodic(grid, pos, mass)
        b, q = t.pm_periodic(grid, pos[:-1], mass[:-1])
        c, _ = t.pm_periodic(grid, pos[:-1], mass[:-1], want_pot=False)
        bad = pos[:-1].copy()
        bad[n // 3, 2] = np.nan
        with pytest.raises(L.GpuGravError) as e:
            t.pm_periodic(grid, bad, mass[:-1])
        assert e.value.status == L.ERR_INVALID
        d, _ = t.pm_periodic(grid, pos[:1], np.ones(1))
    # the deposits of both calls add the same terms in any order: 1e-11 of the largest value
    for x, y in ((a[:-1], b), (p[:-1], q), (c, b)):
        assert np.max(np.abs(x - y)) <= 1e-11 * np.max(np.abs(y))
    assert np.max(np.abs(d)) <= 1e-9  # a lone particle at a mesh point pulls its images only


def test_nonfinite_position_in_brick_order(cuda_lib):
    grid, n = 256, 1 << 23
    rng = np.random.default_rng(10)
    pos, mass = rng.uniform(0, 1, (n, 3)), np.full(n, 1.0 / n)
    asmth = 1.25 / grid
    with GravityTree(L.make_params(periodic=True, box_size=1.0, asmth=asmth, rcut=4.5 * asmth, softening=(1e-3,))) as t:
        a, _ = t.pm_periodic(grid, pos, mass)
        for where, value in ((0, np.nan), (n // 2, np.inf), (n - 1, -1e300)):
            bad = pos.copy()
            bad[where, where % 3] = value
            with pytest.raises(L.GpuGravError) as e:
                t.pm_periodic(grid, bad, mass)
            assert e.value.status == L.ERR_INVALID
        b, _ = t.pm_periodic(grid, pos, mass)
    assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(a))
