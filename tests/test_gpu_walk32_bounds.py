"""Accepted parameters that leave the range the group walk's table was made for, in FP32 and in the walk's FP64
form: particles without softening, which meet their own entry at distance zero (the reference's result for
them is not finite; the others' and the massless ones' are), and an Rcut beyond the table's end."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


def _walk(precision, pos, mass, st, periodic=True, softening=(0.0, 0.01), rcut=4.5 * 0.05, theta=0.0):
    prm = L.make_params(periodic, asmth=0.05 if periodic else 0.0, rcut=rcut if periodic else 0.0, softening=softening,
                        precision=precision, err_tol_theta=theta, err_tol_force_acc=0.0025)
    with GravityTree(prm) as t:
        t.domain_decomposition(pos, mass, st)
        t.construct_forcetree()
        return t.gravity_tree(np.full(len(mass), 0.02, np.float32))


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("precision", [L.PREC_FP32, L.PREC_FP64_GROUP])
@pytest.mark.parametrize("n,theta", [(1999, 0.0), (2000, 0.0), (2000, 0.7), (120003, 0.0)])
@pytest.mark.parametrize("softening", [(0.0, 0.01), (0.0, 0.0)])
def test_particles_without_softening(softening, n, theta, precision, periodic, cuda_lib):
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, 1, (n, 3))
    mass = rng.uniform(0.5, 1.5, n) / n
    st = (np.arange(n) % 3 != 0).astype(np.uint8)  # every third particle is of type 0
    mass[::6] = 0.0  # half of those are massless: no entry of their own
    acc, pot, _ = _walk(precision, pos, mass, st, periodic, softening, theta=theta)
    ok = (mass == 0) | (np.asarray(softening)[st] > 0)
    ref, _, _ = _walk(L.PREC_FP64, pos, mass, st, periodic, softening, theta=theta)
    assert np.array_equal(np.isfinite(ref).all(axis=1), ok)
    assert np.isfinite(acc[ok]).all() and np.isfinite(pot[ok]).all()
    # the group opens at least the nodes that each of its targets does: within the criterion's own error
    scale = np.sqrt(np.mean(np.sum(ref[ok] ** 2, axis=1)))
    assert np.sqrt(np.mean(np.sum((acc - ref)[ok] ** 2, axis=1))) <= 0.03 * scale


@pytest.mark.parametrize("precision", [L.PREC_FP32, L.PREC_FP64_GROUP])
@pytest.mark.parametrize("n,theta", [(2000, 0.0), (2000, 0.7), (120003, 0.0)])
def test_rcut_beyond_the_table(n, theta, precision, cuda_lib):
    """Pairs beyond RcutCells x Asmth contribute nothing, whatever Rcut says."""
    rng = np.random.default_rng(n + 1)
    pos, mass, st = rng.uniform(0, 1, (n, 3)), rng.uniform(0.5, 1.5, n) / n, np.ones(n, np.uint8)
    acc, pot, ni = _walk(precision, pos, mass, st, rcut=1.5 * 4.5 * 0.05, theta=theta)
    one, pot1, ni1 = _walk(precision, pos, mass, st, theta=theta)
    # the same pairs and targets; only nodes whose cell lies between the two radii are visited besides, which
    # changes how the sums are batched
    scale = np.sqrt(np.mean(np.sum(one**2, axis=1)))
    assert np.max(np.linalg.norm(acc - one, axis=1)) <= 1e-5 * scale + 1e-5 * np.max(np.linalg.norm(one, axis=1))
    assert np.max(np.abs(pot - pot1)) <= 1e-5 * np.max(np.abs(pot1))
    assert np.sum(ni != ni1) <= n // 100  # a pair at the table's end may fall on the other side by rounding
