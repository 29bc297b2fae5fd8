"""Working space that a PM call keeps for the next one is given back when another allocation needs it, in the same
context or in another one."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("same", [True, False])
def test_pm_space_is_given_back(same, cuda_lib):
    import torch

    grid, n = 384, 1 << 20  # the records of force and potential take 1.8 GB
    rng = np.random.default_rng(2)
    pos, mass = rng.uniform(0, 1, (n, 3)), np.full(n, 1.0 / n)
    asmth = 1.25 / grid
    prm = L.make_params(periodic=True, box_size=1.0, asmth=asmth, rcut=4.5 * asmth, softening=(1e-3,), precision=L.PREC_FP32)
    ic = ics.grid_box(n1=144, seed=1, pmgrid=288)
    with GravityTree(prm) as pm, GravityTree(ics.params_for(ic, precision=L.PREC_FP32)) as other:
        t = pm if same else other
        a, p = pm.pm_periodic(grid, pos, mass)
        torch.cuda.init()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        fill = torch.empty(free - (400 << 20), dtype=torch.uint8, device="cuda")  # 0.4 GB is left
        try:
            t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])  # takes 0.5 GB
            t.construct_forcetree()
            acc, _, _ = t.gravity_tree()
        finally:
            del fill
            torch.cuda.empty_cache()
        b, q = pm.pm_periodic(grid, pos, mass)
    assert np.isfinite(acc).all()
    assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(a)) and np.max(np.abs(p - q)) <= 1e-11 * np.max(np.abs(p))


def test_group_order_takes_no_space_per_particle(cuda_lib):
    """The relative walk of a clustered set orders its groups in arrays that are there already."""
    import torch

    ic = ics.zoom_box(log2_half=21, seed=3, pmgrid=256)
    n = len(ic["mass"])
    old = np.full(n, 50.0, np.float32)
    prm = ics.params_for(ic, precision=L.PREC_FP32, err_tol_force_acc=0.01)
    with GravityTree(prm) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        t.construct_forcetree()
        t.gravity_tree(old)  # by the geometric criterion: no order
        before, _ = torch.cuda.mem_get_info()
        prm.err_tol_theta = 0.0
        t.set_params(prm)
        t.gravity_tree(old)
        after, _ = torch.cuda.mem_get_info()
    assert before - after <= 4 << 20  # 5 bytes a particle would be 21 MB
