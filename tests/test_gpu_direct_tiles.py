"""The direct sums at the edges of their tiles: gravity_direct around a warp's 32 sources and the switch
from one to four targets per warp (bit-exact with the oracle), and the direct sum of sampled targets
around 32-source tiles, batches of tiles and four-target warps, unsorted and repeated targets, clustered
sources that the short-range form skips by tile (against the oracle's sum of every pair)."""
import numpy as np
import pytest

from arepo_b200 import _lib as L
from arepo_b200 import ics
from arepo_b200.gravity import GravityTree
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _set(kind, n, seed=5):
    rng = np.random.default_rng(seed)
    ic = ics.zoom_box(log2_half=14, seed=seed, pmgrid=48) if kind != "iso" else ics.plummer(max(n, 2), seed=seed)
    keep = rng.permutation(len(ic["mass"]))[:n]
    ic = dict(ic, pos=ic["pos"][keep], mass=ic["mass"][keep], softtype=ic["softtype"][keep])
    if kind == "ewald":
        ic.update(asmth=0.0, rcut=0.0)
    return ic


def _params(ic):
    return (ics.params_for(ic), O.make_params(ic["periodic"], box=ic["box"], asmth=ic["asmth"], rcut=ic["rcut"],
                                              softening=tuple(ic["softening"])))


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("pm", "iso") for n in (2, 31, 32, 33, 129, 8192, 8193)] + [("ewald", 97)])
def test_gravity_direct_tiles(kind, n, cuda_lib):
    ic = _set(kind, n)
    p, op = _params(ic)
    pos = O.wrap(ic["pos"], op)
    a_o, p_o = O.gravity_direct(pos, ic["mass"], ic["softtype"], op)
    with GravityTree(p) as t:
        a, po = t.gravity_direct(pos, ic["mass"], ic["softtype"])
    assert np.array_equal(a, a_o) and np.array_equal(po, p_o)


@pytest.mark.parametrize("kind", ["pm", "iso"])
@pytest.mark.parametrize("n,nt", [(2, 1), (31, 3), (33, 4), (1023, 5), (1025, 64), (20000, 130)])
def test_direct_sum_tiles(kind, n, nt, cuda_lib):
    ic = _set(kind, n)
    p, op = _params(ic)
    tg = np.random.default_rng(7).integers(0, n, nt)
    tg[-1] = tg[0]  # repeated
    with GravityTree(p) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        acc, pot = t.direct(tg)
    acc_o, pot_o = O.direct(O.wrap(ic["pos"], op), ic["mass"], ic["softtype"], op, tg)
    # the two sides' square roots, erfc and exp differ by a few ulp and the pairs are added in another order
    assert np.max(np.abs(acc - acc_o)) < 1e-11 * np.max(np.abs(acc_o))
    assert np.max(np.abs(pot - pot_o)) < 1e-11 * np.max(np.abs(pot_o))


def test_direct_sum_cut_and_scratch(cuda_lib):
    """cut: the pairs inside Rcut only (numpy), and the same results when a larger call came before"""
    ic = _set("pm", 3000)
    p, op = _params(ic)
    pos = O.wrap(ic["pos"], op)
    tg = np.arange(0, 3000, 41)
    with GravityTree(p) as t:
        t.domain_decomposition(ic["pos"], ic["mass"], ic["softtype"])
        a1, p1 = t.direct(tg, cut=True)
        t.direct(np.arange(3000))
        a2, p2 = t.direct(tg, cut=True)
    assert np.array_equal(a1, a2) and np.array_equal(p1, p2)
    from math import erfc

    for k, i in enumerate(tg[:8]):
        d = pos - pos[i]
        d -= np.round(d)
        r = np.sqrt((d * d).sum(1))
        near = (r * r < ic["rcut"] ** 2) & (r > 0)
        h = 2.8 * np.maximum(np.asarray(ic["softening"])[ic["softtype"]], ic["softening"][ic["softtype"][i]])
        far = near & (r >= h)
        u = 0.5 / ic["asmth"] * r[far]
        f = (np.array([erfc(x) for x in u]) + 2 * u / np.sqrt(np.pi) * np.exp(-u * u)) * ic["mass"][far] / r[far] ** 3
        a = (d[far] * f[:, None]).sum(0)
        # softened pairs by the oracle's spline: the particles inside the softening length alone, every pair of
        # which is inside Rcut
        inner = np.append(np.nonzero(near & (r < h))[0], i)
        a_s, _ = O.direct(pos[inner], ic["mass"][inner], ic["softtype"][inner], op, np.array([len(inner) - 1]))
        a += a_s[0]
        assert np.max(np.abs(a - a1[k])) < 1e-11 * np.max(np.abs(a1))
