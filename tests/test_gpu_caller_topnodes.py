"""A caller's TopNodes are checked before particles descend by them: morton_to_peano has to be the curve's, as
domain_determineTopTree writes it (src/domain/domain_toplevel.c:111-269).  A tree whose entries are permuted put
particles below the wrong top nodes."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_FP32])
@pytest.mark.parametrize("mdom", [4, 200])
def test_morton_to_peano_is_checked(mdom, precision, cuda_lib):
    ic = ics.grid_box(n1=14, seed=3, pmgrid=28)
    with GravityTree(ics.params_for(ic, precision=precision, multiple_domains=mdom)) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        top = t.topnodes()
        ref = t.gravity_tree()
        inner = np.nonzero(top["daughter"] >= 0)[0]
        for node in (inner[0], inner[-1]):
            for a, b in ((0, 1), (2, 7)):
                bad = top.copy()
                bad["morton_to_peano"][node][[a, b]] = top["morton_to_peano"][node][[b, a]]
                with pytest.raises(L.GpuGravError) as e:
                    t.construct_forcetree(topnodes=bad)
                assert e.value.status == L.ERR_TOPNODES
        bad = top.copy()
        bad["morton_to_peano"][0][3] = 9
        with pytest.raises(L.GpuGravError):
            t.construct_forcetree(topnodes=bad)
        t.construct_forcetree(topnodes=top)
        for a, b in zip(t.gravity_tree(), ref):
            assert np.array_equal(a, b)
