"""The direct sum of sampled targets deals batches of 4 to 32 source tiles to its warps by the numbers of targets and
tiles; the same targets in calls of other sizes give the same sums up to the order of FP64 additions."""
import numpy as np
import pytest

from arepo_b200 import ics
from arepo_b200.gravity import GravityTree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["zoom", "plummer"])
@pytest.mark.parametrize("n,nt", [(40, 40), (1000, 500), (2000, 500), (2047, 1000), (2049, 130), (16000, 90)])
def test_batches_agree(n, nt, kind, cuda_lib):
    rng = np.random.default_rng(n)
    ic = ics.plummer(n, seed=n) if kind == "plummer" else ics.zoom_box(log2_half=13, seed=7, pmgrid=48)
    keep = rng.permutation(len(ic["mass"]))[:n]
    with GravityTree(ics.params_for(ic)) as t:
        t.domain_decomposition(ic["pos"][keep], ic["mass"][keep], ic["softtype"][keep])
        tg = rng.choice(n, nt, replace=False)
        a, p = t.direct(tg)
        b, q = (np.concatenate(x) for x in zip(*[t.direct(part) for part in np.array_split(tg, 7)]))
    # n terms in any order, most far smaller than the largest sum
    assert np.max(np.linalg.norm(a - b, axis=1)) <= 1e-13 * np.max(np.linalg.norm(a, axis=1))
    assert np.max(np.abs(p - q)) <= 1e-13 * np.max(np.abs(p))
