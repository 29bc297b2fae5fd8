"""The packed evaluation of the FP32 walk (two targets per lane, both halves of a register pair at once) runs where
there are more groups than half the chip's warps; below that every group goes to two warps of one target per lane.
Both do the same operations on the same lists in the same order: a set above the line equals, bit for bit, the sum
of its slices, which lie below it -- with every kind of remainder in the last group, votes in groups that straddle
a core, both criteria, MULTIPLE_NODE_SOFTENING, with and without the potential."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu

LINE = 12 * 148 * 64  # targets up to which a group goes to two warps (24 warps on each of 148 SMs)


@pytest.mark.parametrize("kind,mns", [("plummer", False), ("zoom", False), ("zoom", True), ("grid", False)])
@pytest.mark.parametrize("n", [LINE + 1, LINE + 33, LINE + 63, LINE + 64])
@pytest.mark.parametrize("theta", [0.7, 0.0])
def test_packed_equals_split(kind, mns, n, theta, cuda_lib):
    import torch

    assert torch.cuda.get_device_properties(0).multi_processor_count == 148
    ic = ics.plummer(n, seed=n) if kind == "plummer" else ics.zoom_box(log2_half=16, seed=9, pmgrid=96) if kind == "zoom" else ics.grid_box(
        n1=49, seed=5, pmgrid=98)
    keep = np.random.default_rng(n).permutation(len(ic["mass"]))[:n]
    pos, mass, st = ic["pos"][keep], ic["mass"][keep], ic["softtype"][keep]
    old = np.exp(np.random.default_rng(1).normal(np.log(0.05 if kind == "plummer" else 5.0), 1.0, n)).astype(np.float32)
    with GravityTree(ics.params_for(ic, precision=L.PREC_FP32, err_tol_theta=theta, multiple_node_softening=mns)) as t:
        t.domain_decomposition(pos, mass, st)
        t.construct_forcetree()
        full = t.gravity_tree(old)
        acc, _, ni = t.gravity_tree(old, want_pot=False)
        assert np.array_equal(acc, full[0]) and np.array_equal(ni, full[2])
        for slices in (2, 3):
            parts = [np.zeros_like(x) for x in full]
            for s in range(slices):
                t.set_target_slice(s, slices)
                for p, x in zip(parts, t.gravity_tree(old)):
                    p += x
            for p, x in zip(parts, full):
                assert np.array_equal(p, x)
