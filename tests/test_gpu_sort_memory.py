"""A context whose last set needed the sort by full keys (long runs of equal leading bits) sorts the next one so at
once, and goes back when a set has no such run: the order is the same on every route, for one system and in the
serving loop, and the second load of a clumped set takes one sort less than the first."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200.gravity import GravityTree
from arepo_b200.serving import GravityServer, serving_params

pytestmark = pytest.mark.gpu


def _clumped(n, run, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0, 1, (n, 3))
    if run:
        pos[rng.permutation(n)[:run]] = 0.3 + rng.uniform(0, 3e-8, (run, 3))
    return pos


def _load(t, pos):
    t.domain_decomposition(pos, np.full(len(pos), 1.0 / len(pos)), np.zeros(len(pos), np.uint8))
    return t.timings().sort_ms


@pytest.mark.parametrize("n", [40, 5000])
def test_same_order_on_every_route(n, cuda_lib):
    prm = L.make_params(True, asmth=0.02, rcut=0.09, softening=(1e-3,))
    runs = [0, 33, 33, 32, 33, 0, 0, 35, 2]
    with GravityTree(prm) as one:
        for k, run in enumerate(runs):
            pos = _clumped(n, run, k)
            _load(one, pos)
            with GravityTree(prm) as fresh:
                _load(fresh, pos)
                assert np.array_equal(one.order(), fresh.order())
                for a, b in zip(one.keys(), fresh.keys()):
                    assert np.array_equal(a, b)
            one.construct_forcetree()
            assert np.isfinite(one.gravity_tree()[0]).all()


def test_second_load_sorts_once(cuda_lib):
    n = 1 << 22
    even, clump = _clumped(n, 0, 1), _clumped(n, 100, 1)
    first, second = [], []
    with GravityTree(L.make_params(True, asmth=0.002, rcut=0.009, softening=(1e-4,), precision=L.PREC_FP32)) as t:
        for _ in range(4):
            _load(t, even)
            _load(t, even)
            first.append(_load(t, clump))
            second.append(_load(t, clump))
    assert min(second) < 0.85 * min(first), (first, second)


def test_serving(cuda_lib):
    """systems with and without clumps come and go; each steps as it does alone"""
    rng = np.random.default_rng(4)
    sets = []
    for k in range(6):
        pos = rng.normal(size=(300 + 50 * k, 3))
        if k % 3 == 1:
            pos[:60] = pos[0] + rng.uniform(0, 3e-8, (60, 3))
        sets.append(pos)

    def run(ids, systems):
        with GravityServer(serving_params(0.02), max_systems=systems, max_particles=8192) as srv:
            for k in ids:
                x = sets[k]
                srv.submit(k, x, np.zeros_like(x), np.full(len(x), 1.0 / len(x)), np.zeros(len(x), np.uint8), 1 + k % 3, 0.01)
            return srv.run_to_completion()

    many = run(range(6), 2)
    for k in range(6):
        alone = run([k], 2)[k]
        assert np.array_equal(many[k].pos, alone.pos) and np.array_equal(many[k].acc, alone.acc)
