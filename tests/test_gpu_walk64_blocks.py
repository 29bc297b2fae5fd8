"""The FP64 walk picks its blocks per SM by the number of targets and the depth of the tree: every form gives each
target the same bits, so an even set's walk at the sizes where the choice changes equals the sum of its slices,
which are small enough for the first form."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["pm", "mns", "ewald", "isolated"])
@pytest.mark.parametrize("n1", [49, 50, 56, 58, 65])
def test_forms_agree(n1, form, cuda_lib):
    ic = ics.grid_box(n1=n1, seed=n1, pmgrid=2 * n1)
    n = len(ic["mass"])
    st = (np.arange(n) % 5 == 0).astype(np.uint8)
    pm = form in ("pm", "mns")
    prm = L.make_params(form != "isolated", asmth=ic["asmth"] if pm else 0.0, rcut=ic["rcut"] if pm else 0.0,
                        softening=(1 / 40 / n1, 1 / 10 / n1), precision=L.PREC_FP64, err_tol_theta=0.0, err_tol_force_acc=0.02,
                        multiple_node_softening=form == "mns")
    old = np.full(n, 0.5, np.float32)
    with GravityTree(prm) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], st)
        t.construct_forcetree()
        full = t.gravity_tree(old)
        parts = [np.zeros_like(x) for x in full]
        for s in range(3):
            t.set_target_slice(s, 3)
            for p, x in zip(parts, t.gravity_tree(old)):
                p += x
    for p, x in zip(parts, full):
        assert np.array_equal(p, x)
