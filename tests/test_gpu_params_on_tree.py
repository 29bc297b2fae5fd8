"""Parameters changed on a built tree (gpugrav_set_params keeps the tree when box and softenings stay): each walk
equals that of a context made with those parameters."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [L.PREC_FP32, L.PREC_FP64_GROUP, L.PREC_FP64])
def test_multiple_node_softening_needs_its_tree(precision, cuda_lib):
    ic = ics.zoom_box(log2_half=11, seed=9, pmgrid=32)
    n = len(ic["mass"])
    old = np.full(n, 0.5, np.float32)
    prm = {m: ics.params_for(ic, precision=precision, err_tol_theta=0.0, multiple_node_softening=m) for m in (False, True)}
    ref = {}
    for m in prm:
        with GravityTree(prm[m]) as t:
            t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
            t.construct_forcetree()
            ref[m] = t.gravity_tree(old)
            if m:  # switched off on a tree that has the per-type masses
                t.set_params(prm[False])
                off = t.gravity_tree(old)
    for a, b in zip(off, ref[False]):
        assert np.array_equal(a, b)
    with GravityTree(prm[False]) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        t.set_params(prm[True])
        for call in (lambda: t.gravity_tree(old), lambda: t.gravity_tree_targets(np.arange(5, dtype=np.int32), old), t.mass_per_type):
            with pytest.raises(L.GpuGravError) as e:
                call()
            assert e.value.status == L.ERR_STATE
        t.construct_forcetree()
        for a, b in zip(t.gravity_tree(old), ref[True]):
            assert np.array_equal(a, b)
        assert np.isfinite(t.mass_per_type()).all()


@pytest.mark.parametrize("n1", [9, 20])
def test_split_switched_off_and_on(n1, cuda_lib):
    """TreePM walks two targets per lane, the Ewald walk one: the group table follows."""
    ic = ics.grid_box(n1=n1, seed=44, pmgrid=2 * n1)
    n = len(ic["mass"])
    old = np.full(n, 0.3, np.float32)
    act = np.random.default_rng(1).permutation(n)[: n // 3].astype(np.int32)

    def prm(pm):
        return L.make_params(True, asmth=ic["asmth"] if pm else 0.0, rcut=ic["rcut"] if pm else 0.0, softening=ic["softening"],
                             precision=L.PREC_FP32, err_tol_theta=0.0)

    def walks(t):
        return [*t.gravity_tree(old), *t.gravity_tree_targets(act, old), *t.gravity_tree(old)]

    fresh = {}
    for pm in (True, False):
        with GravityTree(prm(pm)) as t:
            t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
            t.construct_forcetree()
            fresh[pm] = walks(t)
    with GravityTree(prm(True)) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        for pm in (True, False, True):
            t.set_params(prm(pm))
            for a, b in zip(walks(t), fresh[pm]):
                assert np.array_equal(a, b)
