"""Particles that share the leading 64 bits of their Peano-Hilbert keys: short runs are ordered by the full
keys on the spot, longer ones send the whole set through the full sort.  Order, tree and forces stay
bit-exact with the oracle, for one system and in the serving loop."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree
from arepo_b200.serving import GravityServer, serving_params
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _clumps(run, seed=3):
    """a displaced grid with clumps of `run` points closer than the 21st level, and one of identical points"""
    rng = np.random.default_rng(seed)
    ic = ics.grid_box(n1=12, seed=seed, pmgrid=24)
    pos = ic["pos"]
    at = rng.permutation(len(pos))
    for c in range(3):
        pos[at[c * run : (c + 1) * run]] = pos[at[c * run]] + rng.uniform(0, 3e-8, (run, 3))
    pos[at[3 * run : 3 * run + 5]] = pos[at[3 * run]]
    return dict(ic, pos=np.mod(pos, 1.0))


@pytest.mark.parametrize("run", [2, 3, 31, 32, 33, 80])
def test_order_and_forces(run, cuda_lib):
    ic = _clumps(run)
    op = O.make_params(True, box=1.0, asmth=ic["asmth"], rcut=ic["rcut"], softening=tuple(ic["softening"]))
    ref = O.pipeline(ic["pos"], ic["mass"], ic["softtype"], op)
    with GravityTree(ics.params_for(ic)) as t:
        acc, pot, ni, _ = t.compute_grav_accelerations(ic["pos"], ic["mass"], ic["softtype"])
        order = t.order()
        hi, lo = t.keys()
    assert np.array_equal(order, ref["perm"])
    assert np.all((hi[1:] > hi[:-1]) | ((hi[1:] == hi[:-1]) & (lo[1:] >= lo[:-1])))
    assert np.array_equal(acc[order], ref["acc1"]) and np.array_equal(pot[order], ref["pot1"])
    assert np.array_equal(ni[order], ref["ninter1"])


@pytest.mark.parametrize("run", [3, 80])
def test_serving(run, cuda_lib):
    """a system with such clumps steps the same alone and beside others"""
    rng = np.random.default_rng(4)
    pos = rng.normal(size=(500, 3))
    pos[:run] = pos[0] + rng.uniform(0, 3e-8, (run, 3))
    others = [rng.normal(size=(n, 3)) for n in (70, 33)]
    res = []
    for sets in ([pos], [others[0], pos, others[1]]):
        with GravityServer(serving_params(0.02), max_systems=8, max_particles=4096) as srv:
            for k, x in enumerate(sets):
                srv.submit(7 if x is pos else k + 100, x, np.zeros_like(x), np.full(len(x), 1.0 / len(x)), np.zeros(len(x), np.uint8), 2, 0.01)
            res.append(srv.run_to_completion()[7])
    assert np.all(np.isfinite(res[0].acc))
    assert np.array_equal(res[0].pos, res[1].pos) and np.array_equal(res[0].acc, res[1].acc)
