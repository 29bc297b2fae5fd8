"""Target slices of an active list whose groups are cut between distant targets (the background particles on both
sides of a dense core): the slices sum to the unsliced walk, whatever an earlier walk left in the results."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [L.PREC_FP32, L.PREC_FP64_GROUP, L.PREC_FP64])
@pytest.mark.parametrize("every", [1, 7])
def test_slices_of_cut_groups(every, precision, cuda_lib):
    ic = ics.zoom_box(log2_half=14, seed=1004, pmgrid=128)
    n = len(ic["mass"])
    act = np.random.default_rng(6).permutation(np.nonzero(ic["softtype"] == 0)[0][::every]).astype(np.int32)
    old = np.full(n, 0.5, np.float32)
    with GravityTree(ics.params_for(ic, precision=precision, err_tol_theta=0.0)) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        full = t.gravity_tree_targets(act, old)
        for slices in (2, 3, 5):
            parts = [np.zeros_like(x) for x in full]
            for s in range(slices):
                t.set_target_slice(0, 1)
                t.gravity_tree_targets(act, 4 * old)  # other results in the buffers
                t.set_target_slice(s, slices)
                for p, x in zip(parts, t.gravity_tree_targets(act, old)):
                    p += x
            for p, x in zip(parts, full):
                assert np.array_equal(p, x)
