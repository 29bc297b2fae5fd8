"""The group order of isolated sets (the dear half first, the rest by key) and OldAcc values at the ends of its
classes -- zeros, negative and infinite ones, magnitudes beyond the classes: a permutation of the groups whatever
they are, so slices small enough to go in key order sum to the same bits."""
import numpy as np
import pytest

from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plummer", "zoom"])
@pytest.mark.parametrize("values", ["real", "zeros", "one", "huge", "tiny", "odd"])
def test_order_is_a_permutation(values, kind, cuda_lib):
    ic = ics.plummer(500037, seed=4) if kind == "plummer" else ics.zoom_box(log2_half=18, seed=77, pmgrid=128)
    n = len(ic["mass"])
    rng = np.random.default_rng(5)
    old = np.exp(rng.normal(2.0, 2.0, n)).astype(np.float32)
    if values == "zeros":
        old[rng.integers(0, n, 4)] = 0.0
    elif values == "one":
        old[:] = 1.0
    elif values == "huge":
        old[rng.integers(0, n, 40)] = 3e38
    elif values == "tiny":
        old[rng.integers(0, n, 4)] = 1e-44
    elif values == "odd":  # as large as any, to the criterion and to the classes
        old[:64] = np.inf
        old[64:128] = -np.inf
    with GravityTree(ics.params_for(ic, err_tol_theta=0.0, err_tol_force_acc=0.05)) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        assert 8 ** (t.tree_info().max_depth - 9) >= n
        full = t.gravity_tree(old)
        parts = [np.zeros_like(x) for x in full]
        for s in range(8):
            t.set_target_slice(s, 8)
            for p, x in zip(parts, t.gravity_tree(old)):
                p += x
    assert np.all(full[2] > 0)
    for p, x in zip(parts, full):
        assert np.array_equal(p, x)
