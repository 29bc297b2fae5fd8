"""Large sets on large meshes go through the PM in brick order with differences and readout in one pass.  A
set one particle below that line takes the plain path: with a massless last particle both see the same
mesh, and every other particle's result agrees to the rounding of FP64 sums."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,kind", [(256, "even"), (267, "clustered")])
def test_brick_order_against_callers_order(grid, kind, cuda_lib):
    n = 1 << 23
    rng = np.random.default_rng(grid)
    pos = rng.uniform(0, 1, (n, 3))
    if kind == "clustered":
        pos[: n // 2] = (pos[: n // 2] - 0.5) * 0.01 + 0.999  # across the box's faces, into a few bricks
        pos[-1000:] = pos[0]  # many in one cell
    pos[:8] = [[i >> 2, i >> 1 & 1, i & 1] for i in range(8)]  # box corners
    pos[8] = 1.0 - 1e-12
    mass = rng.uniform(0.5, 1.5, n) / n
    mass[-1] = 0.0
    asmth = 1.25 / grid
    with GravityTree(L.make_params(periodic=True, box_size=1.0, asmth=asmth, rcut=4.5 * asmth, softening=(1e-3,))) as t:
        a, p = t.pm_periodic(grid, pos, mass)
        b, q = t.pm_periodic(grid, pos[:-1], mass[:-1])
        c, _ = t.pm_periodic(grid, pos, mass, want_pot=False)
    # sums of up to 4e6 FP64 terms per cell in any order, through the transform: 1e-11 of the largest value
    for x, y in ((a[:-1], b), (p[:-1], q), (c, a)):
        assert np.max(np.abs(x - y)) <= 1e-11 * np.max(np.abs(y))
