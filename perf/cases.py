"""The work a user of this engine has it do, as timed cases.

Each case is one call sequence through the package's public entry points:

  step       one force computation of every particle: domain_decomposition, construct_forcetree,
             gravity_tree (the drop-in for construct_forcetree + gravity_tree of the host code)
  active     the same for the synchronized time bins only: active_particles, gravity_tree_targets
  pm         the periodic long-range force
  serve      a batch of independent systems through the serving loop, submitted, stepped and polled
  forcetest  FP64 direct summation for sampled targets of a loaded set (FORCETEST)
  small      gravity_direct, which replaces the tree below DIRECT_SUMMATION_THRESHOLD particles

Particle sets are those of arepo_b200/ics.py (displaced grid, Hernquist and Plummer spheres, Zel'dovich
box, multi-mass zoom box), drawn on the GPU.  OldAcc, which a running program has from its previous
step, is the smooth acceleration of the set (enclosed mass, or the linear-theory 4 pi G rho psi) plus
the typical pull of a random set's neighbours; "oldacc": "tree" is a program that takes it from the
short-range force alone, as bench.py does, against "total" with the PM force added.
"""
import math

import numpy as np
import torch

from arepo_b200 import _lib as L
from arepo_b200.gravity import GravityTree
from arepo_b200.ics import ASMTH, RCUT
from arepo_b200.serving import GravityServer, serving_params

PRECISION = {"fp32": L.PREC_FP32, "fp64": L.PREC_FP64, "fp64_group": L.PREC_FP64_GROUP}
SERVE_EPS, SERVE_DT = 0.02, 0.005
MAX_PAIRS = 6e10  # pairs that exact() sums within its time


def listed():
    return [
        # a handful of active particles: what gravity() runs instead of the tree
        dict(name="small_1531", kind="small", ic="plummer", n=1531, periodic=False),
        # one small isolated system per call, host arrays: launches and latency
        dict(name="step_plummer_4099", kind="step", ic="plummer", n=4099, precision="fp32", criterion="relative", tol=0.0025, host=True),
        # the bit-exact parity path from AREPO's host arrays, displaced 32^3 grid at PMGRID 64
        dict(name="step64_grid_32", kind="step", ic="grid", n1=32, pmgrid=64, precision="fp64", criterion="relative", tol=0.0025, host=True),
        # the first pass of a run (Barnes-Hut criterion) on an isolated 2^20 Hernquist halo
        dict(name="step_hernquist_bh_2e20", kind="step", ic="hernquist", n=1 << 20, precision="fp32", criterion="bh", tol=0.0025, host=False),
        # a cosmological box early on: few interactions per particle, the build weighs as much as the walk
        dict(name="step_zeldovich_256", kind="step", ic="zeldovich", n1=256, pmgrid=512, precision="fp32", criterion="relative", tol=0.0025, host=False),
        # the benchmark's workload: multi-mass zoom box of 2^24 particles
        dict(name="step_zoom_2e24", kind="step", ic="zoom", n=1 << 24, pmgrid=512, precision="fp32", criterion="relative", tol=6e-5, host=False, oldacc="tree"),
        # parity walk of a clustered two-species set with MULTIPLE_NODE_SOFTENING
        dict(name="step64_zoom_mns_240022", kind="step", ic="zoom", n=240022, pmgrid=128, precision="fp64", criterion="relative", tol=5e-4, host=False, mns=True),
        # hierarchical time stepping: the dense core's time bins are active, host arrays
        dict(name="active_zoom_1000018", kind="active", ic="zoom", n=1000018, pmgrid=256, precision="fp32", tol=6e-5, fraction=0.1),
        # periodic box without PM: Ewald correction per interaction
        dict(name="step_ewald_45", kind="step", ic="grid", n1=45, pmgrid=0, precision="fp32", criterion="relative", tol=0.0025, host=False),
        # the long-range half of the TreePM force of the benchmark's particles
        dict(name="pm_512_2e24", kind="pm", ic="zoom", n=1 << 24, pmgrid=512, host=False),
        # the serving loop on a mix of system sizes
        dict(name="serve_24", kind="serve", systems=24, nmin=1000, nmax=100000, steps=8),
        # accuracy check of a run's forces: exact short-range sum for 4096 targets
        dict(name="forcetest_2e20", kind="forcetest", ic="zoom", n=1 << 20, pmgrid=256, targets=4096, cut=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["step", "active", "pm", "serve", "forcetest", "small"], [50, 10, 14, 8, 10, 8])[0]
    if kind == "small":
        return dict(kind=kind, ic=rng.choice(["plummer", "uniform"]), n=rng.randint(2, 2999), periodic=rng.random() < 0.5)
    if kind == "serve":
        nmin = _log_int(rng, 64, 20000)
        return dict(kind=kind, systems=rng.randint(1, 40), nmin=nmin, nmax=min(200000, nmin * _log_int(rng, 2, 100)), steps=rng.randint(0, 8))
    if kind == "pm":
        n = _log_int(rng, 1000, 1 << 24)
        return dict(kind=kind, ic=rng.choice(["zoom", "uniform"]), n=n, pmgrid=_log_int(rng, 32, 512), host=n < 1 << 20 and rng.random() < 0.5)
    if kind == "active":
        n = _log_int(rng, 4000, 1 << 21)
        return dict(kind=kind, ic="zoom", n=n, pmgrid=max(32, 2 * round(n ** (1 / 3))), precision="fp32" if n > 1 << 17 or rng.random() < 0.7 else "fp64",
                    tol=rng.choice([6e-5, 5e-4, 0.0025]), oldacc=rng.choice(["tree", "total"]), fraction=math.exp(rng.uniform(math.log(0.005), 0.0)))
    if kind == "forcetest":
        n = _log_int(rng, 2000, 1 << 21)
        ic = rng.choice(["zoom", "plummer", "uniform"])
        return dict(kind=kind, ic=ic, n=n, pmgrid=0 if ic == "plummer" else max(32, 2 * round(n ** (1 / 3))), targets=_log_int(rng, 1, 2048),
                    cut=ic != "plummer" and rng.random() < 0.4)
    precision = rng.choices(["fp32", "fp64", "fp64_group"], [70, 20, 10])[0]
    ic = rng.choice(["plummer", "hernquist", "grid", "zeldovich", "zoom"])
    most = {"fp32": 1 << 23, "fp64": 1 << 18, "fp64_group": 1 << 21}[precision]
    n = _log_int(rng, 64, most)
    c = dict(kind=kind, ic=ic, precision=precision, criterion="bh" if rng.random() < 0.2 else "relative", tol=rng.choice([6e-5, 5e-4, 0.0025]),
             host=n < 1 << 20 and rng.random() < 0.5)
    if ic in ("grid", "zeldovich"):
        n1 = max(4, round(n ** (1 / 3)))
        return dict(c, n1=n1, pmgrid=max(8, 2 * n1))
    if ic == "zoom":
        return dict(c, n=n, pmgrid=max(16, 2 * round(n ** (1 / 3))), oldacc=rng.choice(["tree", "total"]), mns=rng.random() < 0.25)
    return dict(c, n=n)


# ---- particle sets -------------------------------------------------------------------------------
def _rand(g, *shape):
    return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=g)


def _normal(g, *shape):
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def _sphere(g, r):
    v = _normal(g, r.numel(), 3)
    return r[:, None] * v / v.norm(dim=1, keepdim=True)


def _plummer(g, n, b, rtrunc=None):
    """positions around the origin and the radii's acceleration per unit mass"""
    umax = 1.0 if rtrunc is None else (1.0 + (b / rtrunc) ** 2) ** -1.5
    u = 1e-12 + (umax - 1e-12) * _rand(g, n)
    r = b / torch.sqrt(u.pow(-2.0 / 3.0) - 1.0)
    return _sphere(g, r), (u / umax) / r**2


def _particles(case, seed):
    """pos, mass, softtype, OldAcc (GPU tensors) and the parameters that go with them"""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    ic, pmgrid = case["ic"], int(case.get("pmgrid", 0))
    periodic = ic in ("grid", "zeldovich", "zoom", "uniform")
    if ic in ("grid", "zeldovich"):
        n1 = int(case["n1"])
        n = n1**3
        ax = (torch.arange(n1, dtype=torch.float64, device="cuda") + 0.5) / n1
        pos = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
        if ic == "grid":
            psi = _normal(g, n, 3) * (0.2 / n1)
            soft = (1 / 40 / n1,)
        else:
            # Gaussian displacements with P(k) ~ k^-2, rms half a grid spacing
            k1 = torch.fft.fftfreq(n1, 1.0 / n1, dtype=torch.float64, device="cuda")
            kz = torch.fft.rfftfreq(n1, 1.0 / n1, dtype=torch.float64, device="cuda")
            kk = torch.meshgrid(k1, k1, kz, indexing="ij")
            k2 = kk[0] ** 2 + kk[1] ** 2 + kk[2] ** 2
            k2[0, 0, 0] = 1.0
            amp = torch.where((kk[0].abs() >= n1 // 2) | (kk[1].abs() >= n1 // 2) | (kk[2].abs() >= n1 // 2), 0.0, k2**-0.5)
            amp[0, 0, 0] = 0.0
            delta = torch.complex(_normal(g, *amp.shape), _normal(g, *amp.shape)) * amp / k2
            psi = torch.stack([torch.fft.irfftn(1j * k * delta, s=(n1, n1, n1), dim=(0, 1, 2)).reshape(-1) for k in kk], 1)
            psi = psi * ((0.5 / n1) / psi.square().sum(1).mean().sqrt())
            soft = (1 / 30 / n1,)
        pos = torch.remainder(pos + psi, 1.0)
        mass = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        st = torch.zeros(n, dtype=torch.uint8, device="cuda")
        old = 4 * math.pi * psi.norm(dim=1)
    elif ic in ("zoom", "uniform"):
        n = int(case["n"])
        nl = n - n // 2 if ic == "zoom" else n
        nh = n - nl
        lo = _rand(g, nl, 3)
        m = 1.0 / (8.0 * nl + nh)
        b = 0.02
        old = torch.full((n,), 2.6 * 8.0 * m * nl ** (2 / 3), dtype=torch.float64, device="cuda")  # neighbours of a random set
        soft = (nl ** (-1 / 3) / 40,)
        pos = lo
        if nh:
            hi, a = _plummer(g, nh, b, 0.1)
            pos = torch.cat([lo, torch.remainder(0.5 + hi, 1.0)])
            r2 = (lo - 0.5).square().sum(1)
            inside = torch.clamp((r2 / (r2 + b * b)).pow(1.5) * (1.0 + (b / 0.1) ** 2) ** 1.5, max=1.0)
            if case.get("oldacc") == "tree":
                # the part of a smooth density within a few Asmth: 4 pi Asmth^2 |grad rho|
                rr = (pos[nl:] - 0.5).norm(dim=1)
                smooth = 15 * nh * m * (ASMTH / pmgrid) ** 2 / b**3 * rr / (rr**2 + b * b) * (1 + rr**2 / b**2) ** -2.5
                near = 2.6 * m ** (1 / 3) * (3 * nh * m / (4 * math.pi * b**3)) ** (2 / 3) * (1 + rr**2 / b**2) ** (-5 / 3)
                old[nl:] = torch.hypot(smooth, near)
            else:
                old = torch.hypot(old, torch.cat([nh * m * inside / r2, nh * m * a]))
            soft += ((4 / 3 * math.pi * (1.305 * b) ** 3 / (nh / 2)) ** (1 / 3) / 40,)
        mass = torch.cat([torch.full((nl,), 8.0 * m, dtype=torch.float64, device="cuda"), torch.full((nh,), m, dtype=torch.float64, device="cuda")])
        st = torch.cat([torch.zeros(nl, dtype=torch.uint8, device="cuda"), torch.ones(nh, dtype=torch.uint8, device="cuda")])
    else:
        n = int(case["n"])
        if ic == "plummer":
            pos, old = _plummer(g, n, 1.0)
            soft = (0.02,)
        else:
            su = torch.sqrt(_rand(g, n) * (50.0 / 51.0) ** 2)
            r = su / (1.0 - su)
            pos = _sphere(g, r)
            old = 1.0 / (1.0 + r) ** 2
            soft = (0.01,)
        mass = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        st = torch.zeros(n, dtype=torch.uint8, device="cuda")
    asmth = ASMTH / pmgrid if pmgrid else 0.0
    return dict(pos=pos.contiguous(), mass=mass, st=st, old=old.to(torch.float32), soft=soft, periodic=periodic, asmth=asmth, rcut=RCUT * asmth)


def _small(case, seed):
    c = dict(case)
    if c["periodic"]:
        c["pmgrid"] = 16
    d = _particles(c, seed)
    if c["periodic"] and c["ic"] == "plummer":
        d["pos"] = torch.remainder(0.5 + 0.05 * d["pos"], 1.0)
        d["soft"] = (0.001,)
    if not c["periodic"]:
        d["asmth"] = d["rcut"] = 0.0
    return dict(d, periodic=bool(c["periodic"]))


def _params(d, case):
    return L.make_params(d["periodic"], asmth=d["asmth"], rcut=d["rcut"], rcut_cells=RCUT, softening=d["soft"],
                         err_tol_theta=0.7 if case.get("criterion") == "bh" else 0.0, err_tol_force_acc=case.get("tol", 0.0025),
                         precision=PRECISION[case.get("precision", "fp32")], multiple_node_softening=bool(case.get("mns", False)))


def _systems(case, seed):
    """sizes (log-uniform) and particle sets of a serving batch, half Plummer and half Hernquist"""
    rng = np.random.default_rng(1005)  # the sizes belong to the case, the particles to the seed
    ns = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1), int(case["systems"]))).astype(np.int64)
    return [_particles(dict(ic=("plummer", "hernquist")[i % 2], n=int(n)), 1000 * int(seed) + i) for i, n in enumerate(ns)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        sets = _systems(case, seed)
        sys = [(s["pos"].cpu().numpy(), np.zeros((len(s["pos"]), 3)), s["mass"].cpu().numpy(), s["st"].cpu().numpy()) for s in sets]
        total = sum(len(s[2]) for s in sys)
        out = {k: np.zeros((total, 3)) for k in ("pos", "vel", "acc")}
        at = np.concatenate([[0], np.cumsum([len(s[2]) for s in sys])])
        bufs = {i: tuple(out[k][at[i] : at[i + 1]] for k in ("pos", "vel", "acc")) for i in range(len(sys))}
        srv = GravityServer(serving_params(SERVE_EPS), max_systems=64, max_particles=max(64, total))
        return dict(kind=kind, srv=srv, sys=sys, out=out, bufs=bufs, steps=int(case["steps"]))
    d = _small(case, seed) if kind == "small" else _particles(case, seed)
    s = dict(kind=kind, case=case, tree=GravityTree(_params(d, case)))
    host = kind in ("small", "active") or bool(case.get("host", False))
    for k in ("pos", "mass", "st", "old"):
        s[k] = d[k].cpu().numpy() if host else d[k]
    s["mem"] = L.MEM_HOST if host else L.MEM_DEVICE
    if not host:
        s["tree"].set_stream(torch.cuda.current_stream().cuda_stream)
    n = len(s["mass"])
    if kind == "step" and not host:
        s["out"] = (torch.empty(n, 3, dtype=torch.float64, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda"),
                    torch.empty(n, dtype=torch.int32, device="cuda"))
    if kind == "active":
        # the particles with the largest accelerations are on the shorter steps: time bin 20 of 30
        s["bins"] = np.full(n, 24, np.int8)
        s["bins"][np.argsort(s["old"], kind="stable")[n - max(1, int(n * case["fraction"])) :]] = 20
        s["sync"] = [b <= 20 for b in range(64)]
    if kind == "forcetest":
        s["tree"].domain_decomposition(s["pos"], s["mass"], s["st"], mem=s["mem"])
        s["targets"] = np.sort(np.random.default_rng(int(seed)).choice(n, min(n, int(case["targets"])), replace=False))
    return s


def run(s):
    kind = s["kind"]
    if kind == "serve":
        srv = s["srv"]
        for i, (pos, vel, mass, st) in enumerate(s["sys"]):
            srv.submit(i, pos, vel, mass, st, nsteps=s["steps"], dt=SERVE_DT)
        while srv.busy():
            srv.tick()
            srv.poll_all(s["bufs"])
        return s["out"]
    t = s["tree"]
    if kind == "small":
        return t.gravity_direct(s["pos"], s["mass"], s["st"])
    if kind == "pm":
        return t.pm_periodic(int(s["case"]["pmgrid"]), s["pos"], s["mass"], mem=s["mem"])
    if kind == "forcetest":
        return t.direct(s["targets"], cut=bool(s["case"]["cut"]))
    t.domain_decomposition(s["pos"], s["mass"], s["st"], mem=s["mem"])
    t.construct_forcetree()
    if kind == "active":
        targets = t.active_particles(s["bins"], s["sync"])
        return (targets, *t.gravity_tree_targets(targets, s["old"]))
    if s["mem"] == L.MEM_HOST:
        return t.gravity_tree(s["old"])
    return t.gravity_tree(s["old"], *s["out"], mem=s["mem"])


# ---- what a pass cannot do without ----------------------------------------------------------------
def _count(case):
    return int(case["n1"]) ** 3 if "n1" in case else int(case["n"])


def _interactions(case):
    """interactions per target of the tree walk, as measured within a factor of about two"""
    n, ic = _count(case), case["ic"]
    tight = 1.0 if case.get("criterion") == "bh" else (0.0025 / case.get("tol", 0.0025)) ** 0.4
    if ic in ("grid", "zeldovich") and case.get("pmgrid"):
        return min(n, 100 * tight)
    if ic == "zoom":
        return min(n, 150 * (n / 4096) ** 0.3 * tight)
    if ic in ("grid", "zeldovich"):
        return min(n, 8000 * tight)
    return min(n, 180 * math.log2(n / 32 + 2) * tight)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        n = case["systems"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        force = min(n, 1500)
        return {"bytes": 57 * n + 72 * n, "flops": (case["steps"] + 2) * 23 * force * n}
    n = _count(case)
    if kind == "small":
        return {"bytes": 33 * n + 32 * n, "flops": 23 * n * n}
    if kind == "pm":
        g = int(case["pmgrid"])
        return {"bytes": 32 * n + 32 * n, "flops": 2 * 2.5 * g**3 * math.log2(g**3) + 100 * n}
    if kind == "forcetest":
        # the factor vanishes in double precision beyond 13 Asmth
        near = 13 * ASMTH / case["pmgrid"] if case["pmgrid"] else 1.0
        share = min(1.0, 4.2 * near**3 + (0.5 if case["ic"] == "zoom" else 0.0)) if case["pmgrid"] else 1.0
        return {"bytes": 33 * n + 40 * case["targets"], "flops": 23 * share * n * case["targets"]}
    targets = n * case["fraction"] if kind == "active" else n
    return {"bytes": 37 * n + 36 * targets, "flops": 23 * _interactions(case) * targets}


# ---- the same results in 64 bits, by direct summation and numpy-style transforms -------------------
def _table(rcut_cells=RCUT, ntab=127):
    """the short-range factors of the TreePM split as the code tabulates them (float entries)"""
    u = torch.arange(ntab + 1, dtype=torch.float64, device="cuda") * (rcut_cells / 2 / ntab)
    force = (torch.erfc(u) + 2 * u / math.sqrt(math.pi) * torch.exp(-u * u) - 1) / torch.where(u > 0, u * u, 1.0)
    force[0] = 0.0
    return force.float().double(), -torch.erfc(u).float().double()


def _pairs(tpos, th, pos, mass, h, periodic, asmth, mode):
    """accelerations and potentials of targets, summed over every source; mode "table": the tree's tabulated
    short-range factor inside its table, "full": the exact factor of every pair, "cut": inside Rcut"""
    acc, pot = torch.zeros_like(tpos), torch.zeros(len(tpos), dtype=torch.float64, device="cuda")
    step = max(1, 20_000_000 // len(pos))
    ft, pt = _table() if asmth else (None, None)
    for a in range(0, len(tpos), step):
        d = [pos[None, :, k] - tpos[a : a + step, k, None] for k in range(3)]
        if periodic:
            d = [x - torch.round(x) for x in d]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        r = torch.sqrt(r2)
        hm = torch.maximum(th[a : a + step, None], h[None, :])
        ri = torch.where(r > 0, 1.0 / r, 0.0)
        fac, wp = ri * ri * ri, -ri
        soft = (r < hm).nonzero(as_tuple=True)
        if len(soft[0]):
            hi = 1.0 / hm[soft]
            u = r[soft] * hi
            u2, u3 = u * u, u**3
            ui = torch.where(u > 0, 1 / u, 0.0)
            near = u < 0.5
            fac[soft] = hi**3 * torch.where(near, 32 / 3 + u2 * (32 * u - 38.4), 64 / 3 - 48 * u + 38.4 * u2 - 32 / 3 * u3 - ui**3 / 15)
            wp[soft] = hi * torch.where(near, -2.8 + u2 * (16 / 3 + u2 * (6.4 * u - 9.6)),
                                        -3.2 + ui / 15 + u2 * (32 / 3 + u * (-16 + u * (9.6 - 32 / 15 * u))))
        if asmth and mode == "table":
            te = r * (0.5 / asmth * (127 / (RCUT / 2)))
            i = te.long()
            inside = i < 127
            i = torch.clamp(i, max=126)
            x = te - i
            fac = torch.where(inside, fac + ri * (0.25 / asmth**2) * ((1 - x) * ft[i] + x * ft[i + 1]), 0.0)
            wp = torch.where(inside, wp + ri * (1 + (1 - x) * pt[i] + x * pt[i + 1]), 0.0)
        elif asmth:
            u = 0.5 / asmth * r
            e = torch.erfc(u)
            fac = fac + ri**3 * (e + 2 / math.sqrt(math.pi) * u * torch.exp(-u * u) - 1)
            wp = wp - ri * (e - 1)
            if mode == "cut":
                inside = r2 < (RCUT * asmth) ** 2
                fac, wp = torch.where(inside, fac, 0.0), torch.where(inside, wp, 0.0)
        fac = fac * mass
        for k in range(3):
            acc[a : a + step, k] = (d[k] * fac).sum(1)
        pot[a : a + step] = (wp * mass).sum(1)
    return acc, pot


def _exact_pm(d, n):
    """CIC mesh, Green's function with deconvolution, 4-point differences and CIC readout"""
    pos, mass = d["pos"], d["mass"]
    xs = pos * n
    i0 = torch.floor(xs)
    w1 = xs - i0
    i0 = torch.remainder(i0.long(), n)
    i1 = torch.remainder(i0 + 1, n)
    nodes = [(ix, iy, iz) for ix in (0, 1) for iy in (0, 1) for iz in (0, 1)]

    def at(q):
        idx = [(i1 if q[k] else i0)[:, k] for k in range(3)]
        w = [(w1 if q[k] else 1 - w1)[:, k] for k in range(3)]
        return (idx[0] * n + idx[1]) * n + idx[2], w[0] * w[1] * w[2]

    rho = torch.zeros(n**3, dtype=torch.float64, device="cuda")
    for q in nodes:
        c, w = at(q)
        rho.index_add_(0, c, w * mass)
    rk = torch.fft.rfftn(rho.view(n, n, n))
    del rho
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    k = 2 * math.pi * torch.where(i >= n // 2, i - n, i)
    s = torch.where(k == 0, 1.0, torch.sin(k / (2 * n)) / torch.where(k == 0, 1.0, k / (2 * n)))
    ax = torch.exp(-k * k * d["asmth"] ** 2) / s**4
    nz = n // 2 + 1
    k2 = (k * k)[:, None, None] + (k * k)[None, :, None] + (k * k)[None, None, :nz]
    k2[0, 0, 0] = 1.0
    for x in range(n):
        rk[x] *= -(ax[x] * ax[:, None] * ax[None, :nz]) / k2[x]
    rk[0, 0, 0] = 0
    del k2
    phi = torch.fft.irfftn(rk, s=(n, n, n)) * (4 * math.pi * float(n) ** 3)
    del rk
    acc = torch.zeros_like(pos)
    pot = torch.zeros(len(pos), dtype=torch.float64, device="cuda")
    for dim in range(-1, 3):
        mesh = phi if dim < 0 else (4 / 3 * (phi.roll(1, dim) - phi.roll(-1, dim)) - 1 / 6 * (phi.roll(2, dim) - phi.roll(-2, dim))) * (n / 2)
        flat = mesh.reshape(-1)
        for q in nodes:
            c, w = at(q)
            if dim < 0:
                pot += flat[c] * w
            else:
                acc[:, dim] += flat[c] * w
    return acc, pot


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        sets = _systems(case, seed)
        if sum(len(s["mass"]) ** 2 for s in sets) * (case["steps"] + 1) > MAX_PAIRS:
            return None
        out = {"pos": [], "vel": [], "acc": []}
        for s in sets:
            h = torch.full_like(s["mass"], 2.8 * SERVE_EPS)
            x, v = s["pos"].clone(), torch.zeros_like(s["pos"])
            force = lambda x: _pairs(x, h, x, s["mass"], h, False, 0.0, "full")[0]  # noqa: E731
            a = force(x)
            for _ in range(int(case["steps"])):
                v = v + 0.5 * SERVE_DT * a
                x = x + SERVE_DT * v
                a = force(x)
                v = v + 0.5 * SERVE_DT * a
            for k, y in (("pos", x), ("vel", v), ("acc", a)):
                out[k].append(y.cpu().numpy())
        return {k: np.concatenate(v) for k, v in out.items()}
    n = _count(case)
    if kind == "pm":
        return _exact_pm(_particles(case, seed), int(case["pmgrid"]))
    d = _small(case, seed) if kind == "small" else _particles(case, seed)
    h = 2.8 * torch.tensor(d["soft"], dtype=torch.float64, device="cuda")[d["st"].long()]
    targets = torch.arange(n, device="cuda")
    if kind == "forcetest":
        targets = torch.from_numpy(np.sort(np.random.default_rng(int(seed)).choice(n, min(n, int(case["targets"])), replace=False))).cuda()
    if len(targets) * n > MAX_PAIRS or kind == "active" or (d["periodic"] and not d["asmth"]):
        return None
    mode = ("cut" if case["cut"] else "full") if kind == "forcetest" else "table"
    acc, pot = _pairs(d["pos"][targets], h[targets], d["pos"], d["mass"], h, d["periodic"], d["asmth"], mode)
    acc, pot = (acc.cpu().numpy(), pot.cpu().numpy()) if kind != "step" or case["host"] else (acc, pot)
    return (acc, pot) if kind != "step" else (acc, pot, None)
