"""Every transfer of the library goes on the stream whose kernels read it.  The contexts' streams are
non-blocking: they do not wait for the default stream, and a plain cudaMemcpy of pageable memory may return
before its last piece has arrived."""
import glob
import os
import re

import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200.gravity import GravityTree
from oracle import oracle as O

CSRC = os.path.join(os.path.dirname(os.path.abspath(L.__file__)), "csrc")


def test_no_transfer_on_the_default_stream():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"#ifdef GG_WALK32_STATS.*?#endif", "", open(path).read(), flags=re.S)  # measurement builds
        text = re.sub(r"//[^\n]*", "", text)
        found += [os.path.basename(path) + ": " + m for m in re.findall(r"\bcuda(?:Memcpy|Memset|MemcpyToSymbol|MemcpyFromSymbol)\(", text)]
    assert not found, found


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [L.PREC_FP32, L.PREC_FP64])
def test_replaced_ewald_tables(precision, cuda_lib):
    """Tables replaced on a live context: every walk sees the whole of the tables last set."""
    rng = np.random.default_rng(8)
    n = 3000
    pos, mass, st = rng.uniform(0, 2.0, (n, 3)), np.full(n, 1.0 / n), np.zeros(n, np.uint8)
    t0 = O.ewald_table()
    old = np.full(n, 0.5, np.float32)
    prm = L.make_params(periodic=True, box_size=2.0, asmth=0.0, rcut=0.0, softening=(0.004,), precision=precision, err_tol_theta=0.0)

    def walk(t, f):
        t.set_ewald_table(*[f * x for x in t0])
        return t.gravity_tree(old)

    with GravityTree(prm) as a:
        a.domain_decomposition(pos, mass, st)
        a.construct_forcetree()
        seen = {f: walk(a, f) for f in (0.25, 0.0, 0.5)}
        for f in (0.5, 0.25, 0.0, 0.25):
            for x, y in zip(walk(a, f), seen[f]):
                assert np.array_equal(x, y)
    # the correction enters linearly: 0.25 and 0.5 times the tables lie on one line with none
    for k in (0, 1):
        d1, d2 = seen[0.25][k] - seen[0.0][k], seen[0.5][k] - seen[0.0][k]
        scale = np.max(np.abs(seen[0.0][k]))
        tol = (1e-11 if precision == L.PREC_FP64 else 1e-4) * scale
        assert np.max(np.abs(d2 - 2 * d1)) <= tol and np.max(np.abs(d1)) > 10 * tol
