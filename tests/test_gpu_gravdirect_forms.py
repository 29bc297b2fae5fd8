"""gravity_direct takes one of three forms by the number of particles; all add the same terms in the same order.  A
massless particle at the end takes a set over the line to the next form and adds nothing to the others' sums: the
results of both sides of each line agree bit for bit."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("iso", 8192), ("pm", 8192), ("ewald", 8192), ("iso", 45000), ("pm", 45000), ("ewald", 110000)])
def test_forms_agree(kind, n, cuda_lib):
    rng = np.random.default_rng(n)
    pos, mass, st = rng.uniform(0, 1, (n + 1, 3)), rng.uniform(0.5, 1.5, n + 1) / n, (rng.uniform(size=n + 1) < 0.3).astype(np.uint8)
    pos[1] = pos[0]
    mass[-1] = 0.0
    prm = L.make_params(kind != "iso", asmth=0.05 if kind == "pm" else 0.0, rcut=0.225 if kind == "pm" else 0.0, softening=(0.001, 0.01))
    with GravityTree(prm) as t:
        a, p = t.gravity_direct(pos[:n], mass[:n], st[:n])
        b, q = t.gravity_direct(pos, mass, st)
        c, _ = t.gravity_direct(pos, mass, st, want_pot=False)
        st[n // 2] = 2
        with pytest.raises(L.GpuGravError) as e:
            t.gravity_direct(pos, mass, st)
        assert e.value.status == L.ERR_INVALID
    assert np.isfinite(b).all() and np.isfinite(q).all()
    assert np.array_equal(a, b[:n]) and np.array_equal(p, q[:n]) and np.array_equal(b, c)
