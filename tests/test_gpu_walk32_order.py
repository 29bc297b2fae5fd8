"""The FP32 walk's groups in order of falling cost (relative criterion, clustered sets of more groups than
resident warps): a group's result is its own, so the walk in this order, by slices of equal size and of equal
cost, equals the same walk by slices small enough to go in key order, bit for bit."""
import numpy as np
import pytest

from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zeros", [0, 5])
def test_group_order_changes_nothing(zeros, cuda_lib):
    ic = ics.zoom_box(log2_half=18, seed=77, pmgrid=128)
    n = len(ic["mass"]) - 37  # the last group and the last run of groups are not full
    ic = dict(ic, pos=ic["pos"][:n], mass=ic["mass"][:n], softtype=ic["softtype"][:n])
    rng = np.random.default_rng(5)
    oldacc = np.exp(rng.normal(6.0, 2.0, n)).astype(np.float32)
    oldacc[rng.integers(0, n, zeros)] = 0  # these open every node inside Rcut
    cost = np.exp(rng.normal(0.0, 2.0, n)).astype(np.float32)
    with GravityTree(ics.params_for(ic, err_tol_theta=0.0)) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        assert 8 ** (t.tree_info().max_depth - 4) >= n and n > 2 * 64 * 3552
        full = t.gravity_tree(oldacc)

        def by_slices(count, cost=None):
            parts = [np.zeros_like(x) for x in full]
            for s in range(count):
                t.set_target_slice(s, count) if cost is None else t.set_target_slice_cost(s, count, cost)
                for p, x in zip(parts, t.gravity_tree(oldacc)):
                    p += x
            t.set_target_slice(0, 1)
            return parts

        small = by_slices(8)
        for other in (full, by_slices(2), by_slices(2, cost)):
            for a, b in zip(small, other):
                assert np.array_equal(a, b)
