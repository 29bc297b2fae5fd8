"""The FP64 walk takes 4 to 32 targets per warp by the number of targets; every target steps through its own
sequence, so the walk by slices (fewer targets per warp) equals the whole one bit for bit, and a small set
equals the same targets of an active list."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,mns", [("plummer", 3, False), ("plummer", 14209, False), ("zoom", 32767, True), ("zoom", 60001, False),
                                        ("plummer", 120001, False)])
def test_targets_per_warp_change_nothing(kind, n, mns, cuda_lib):
    ic = ics.plummer(n, seed=n) if kind == "plummer" else ics.zoom_box(log2_half=15, seed=3, pmgrid=64)
    ic = dict(ic, pos=ic["pos"][:n], mass=ic["mass"][:n], softtype=ic["softtype"][:n])
    n = len(ic["mass"])
    old = np.full(n, 0.05 if kind == "plummer" else 50.0, np.float32)
    with GravityTree(ics.params_for(ic, precision=L.PREC_FP64, err_tol_theta=0.0, multiple_node_softening=mns)) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        full = t.gravity_tree(old)
        parts = [np.zeros_like(x) for x in full]
        for s in range(7):
            t.set_target_slice(s, 7)
            for p, x in zip(parts, t.gravity_tree(old)):
                p += x
        t.set_target_slice(0, 1)
        few = np.arange(0, n, 3, dtype=np.int32)
        act = t.gravity_tree_targets(few, old)
    for a, b, c in zip(full, parts, act):
        assert np.array_equal(a, b)
        assert np.array_equal(a[few], c)
