"""The FP32 group walk at its edges: groups of 64 with every kind of remainder, blocks of list entries,
sets whose groups straddle a core (per-target votes), both criteria, with and without the potential and
MULTIPLE_NODE_SOFTENING.  Its packed evaluation does the scalar one's operations, so against the same
groups in FP64 arithmetic the interaction counts agree and the forces differ by FP32 rounding only."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


def _set(kind, n):
    rng = np.random.default_rng(n)
    ic = ics.plummer(max(n, 2), seed=n) if kind == "plummer" else ics.zoom_box(log2_half=13, seed=9, pmgrid=32)
    keep = rng.permutation(len(ic["mass"]))[:n]
    return dict(ic, pos=ic["pos"][keep], mass=ic["mass"][keep], softtype=ic["softtype"][keep])


@pytest.mark.parametrize("kind,mns", [("plummer", False), ("zoom", False), ("zoom", True)])
@pytest.mark.parametrize("n", [2, 31, 63, 64, 65, 129, 3001, 9999])
@pytest.mark.parametrize("theta", [0.7, 0.0])
def test_packed_against_fp64_arithmetic(kind, mns, n, theta, cuda_lib):
    ic = _set(kind, n)
    old = np.full(n, 0.05 if kind == "plummer" else 0.5, np.float32)
    out = {}
    for prec in (L.PREC_FP32, L.PREC_FP64_GROUP):
        with GravityTree(ics.params_for(ic, precision=prec, err_tol_theta=theta, multiple_node_softening=mns)) as t:
            t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
            t.construct_forcetree()
            out[prec] = t.gravity_tree(old)
            acc, _, ni = t.gravity_tree(old, want_pot=False)
            assert np.array_equal(acc, out[prec][0]) and np.array_equal(ni, out[prec][2])
    a, b = out[L.PREC_FP32], out[L.PREC_FP64_GROUP]
    scale = np.sqrt(np.mean(np.sum(b[0] ** 2, axis=1)))
    # one FP32 rounding per operation and batch sums of up to 256 terms
    assert np.sqrt(np.mean(np.sum((a[0] - b[0]) ** 2, axis=1))) <= 1e-5 * scale
    assert np.max(np.abs(a[1] - b[1])) <= 1e-5 * np.max(np.abs(b[1]))
    # a pair may fall on the other side of Rcut by rounding
    assert np.sum(a[2] != b[2]) <= (0 if kind == "plummer" else max(1, n // 1000))
