"""Performance cases of the GPU solvers.

Each case is one call that a program built on this package makes over and over:
a 3D Newton solve, a forest of 3D systems, a batch of 2D systems, or a short
stream through the request loop.  ``listed`` gives the fixed cases, ``draw``
more of the same ranges.

Ranges: 3D solves of 1e3 to 4e6 particles (uniform, Plummer, Gaussian blobs),
orders 4 to 16 in mixed precision and 6 to 20 in FP64, leaf capacities 20 to
96, rotate and kkylin translations, potential alone or with the field, device
or host arrays; forests of 8 to 96 systems; 2D batches of 1 to 256 systems at
order 20; request streams over the three tolerances of the serving
configuration.

A mixed-precision solve computes in single precision and stores its sums in
doubles; the program that asks for one uses the result in single precision,
so those cases return float32.  FP64 solves return what the solver wrote.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import aran_gb300

ORDERS_MIXED = (4, 6, 8, 10, 12, 16)
ORDERS_FP64 = (6, 8, 10, 12, 16, 20)
LEAVES = (20, 32, 64, 96)
TOLERANCES = (1e-4, 1e-6, 1e-9)


def _solve(name, dist, n, order, maxbox=64, precision="mixed", flavour="rotate", field=True,
           host=False):
    return dict(name=name, kind="solve3d", dist=dist, n=n, order=order, maxbox=maxbox,
                precision=precision, flavour=flavour, field=field, host=host)


def listed():
    return [
        # the smallest everyday solve (C1): latency and launches count
        _solve("uniform10k_p8_pot", "uniform", 10_000, 8, maxbox=20, field=False),
        # the clustered headline set, a simulation step at the usual order
        _solve("plummer4m_p12", "plummer", 4_000_000, 12),
        # the same set where 1e-6 is asked for: the high mixed order
        _solve("plummer4m_p16", "plummer", 4_000_000, 16),
        # a mid-size clustered step at high order, ragged size
        _solve("plummer150k_p16", "plummer", 149_987, 16),
        # a mid-size step at low order on blobs, ragged size
        _solve("blobs300k_p8", "blobs", 299_993, 8),
        # a program on host arrays (copies counted) with smaller leaves, served order
        _solve("uniform131k_p10_host", "uniform", 131_071, 10, maxbox=32, host=True),
        # the plain double-precision path
        _solve("plummer200k_p12_fp64", "plummer", 200_000, 12, precision="fp64"),
        # the second translation family
        _solve("uniform200k_p12_kkylin", "uniform", 200_003, 12, flavour="kkylin"),
        # many independent small systems in one call (C4, 3D)
        dict(name="forest48_p4", kind="forest3d", sizes=1, systems=48, nlo=1000, nhi=100_000,
             order=4, maxbox=64, precision="mixed", field=True),
        # many independent 2D systems in one call (C4, 2D)
        dict(name="batch2d_128_mixed", kind="batch2d", sizes=1, systems=128, nlo=1000, nhi=60_000,
             order=20, maxbox=32, precision="mixed"),
        # one 2D system in double precision (the dummypot program)
        dict(name="plane60k_fp64", kind="batch2d", sizes=1, systems=1, nlo=60_000, nhi=60_000,
             order=20, maxbox=32, precision="fp64"),
        # concurrent requests that name a tolerance (C5)
        dict(name="served8", kind="served", sizes=1, requests=8, nlo=1000, nhi=60_000, slots=4),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(("solve3d",) * 6 + ("fp64", "kkylin", "forest3d", "batch2d", "served"))
    if what in ("solve3d", "fp64", "kkylin"):
        precision = "fp64" if what == "fp64" else "mixed"
        order = rng.choice(ORDERS_FP64 if what == "fp64" else ORDERS_MIXED)
        if what == "fp64":
            top = 400_000 if order <= 12 else 60_000
        elif what == "kkylin":
            top = 500_000 if order <= 12 else 100_000
        else:
            top = 3_000_000
        return dict(kind="solve3d", dist=rng.choice(("uniform", "plummer", "blobs")),
                    n=_logu(rng, 1000, top), order=order, maxbox=rng.choice(LEAVES),
                    precision=precision, flavour="kkylin" if what == "kkylin" else "rotate",
                    field=rng.random() < 0.8, host=rng.random() < 0.25)
    if what == "forest3d":
        return dict(kind="forest3d", sizes=rng.randint(2, 1 << 20), systems=_logu(rng, 8, 96),
                    nlo=1000, nhi=_logu(rng, 5000, 100_000), order=rng.choice((4, 8, 12)),
                    maxbox=64, precision="mixed", field=True)
    if what == "batch2d":
        precision = rng.choice(("mixed", "fp64"))
        systems = _logu(rng, 1, 256 if precision == "mixed" else 16)
        return dict(kind="batch2d", sizes=rng.randint(2, 1 << 20), systems=systems, nlo=1000,
                    nhi=_logu(rng, 2000, 60_000), order=20, maxbox=rng.choice((20, 32, 64)),
                    precision=precision)
    return dict(kind="served", sizes=rng.randint(2, 1 << 20), requests=rng.randint(4, 10),
                nlo=1000, nhi=_logu(rng, 5000, 60_000), slots=rng.choice((2, 4)))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _u(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _points(dist, n, g):
    """Positions, charges and the box of a 3D set (distributions of
    aran_gb300.workloads, drawn on the GPU)."""
    if dist == "uniform":
        return _u(g, n, 3), 2 * _u(g, n) - 1, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)
    if dist == "plummer":
        a = 0.05
        # inverse sampling of the cumulative mass up to the radial cut r = 1
        x1 = (1e-12 + (1 - 1e-12) * _u(g, n)) * (1 + a * a) ** -1.5
        r = a / torch.sqrt(x1 ** (-2.0 / 3.0) - 1)
        z = (1 - 2 * _u(g, n)) * r
        t = torch.sqrt(torch.clamp(r * r - z * z, min=0))
        f = 2 * math.pi * _u(g, n)
        x = torch.stack([t * torch.cos(f), t * torch.sin(f), z], dim=1).contiguous()
        return x, _u(g, n), (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)
    k = 1 + int(torch.randint(0, 8, (1,), generator=g, device="cuda"))
    centres, sig = 0.2 + 0.6 * _u(g, k, 3), 0.02 + 0.18 * _u(g, k)
    which = torch.randint(0, k, (n,), generator=g, device="cuda")
    x = centres[which] + sig[which, None] * torch.randn(n, 3, generator=g, device="cuda",
                                                        dtype=torch.float64)
    x.clamp_(0.0, math.nextafter(1.0, 0.0))
    return x, 2 * _u(g, n) - 1, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)


def _sizes(case, count):
    """Log-uniform system sizes: part of the case, not of the seed."""
    r = random.Random(case["sizes"])
    return [_logu(r, case["nlo"], case["nhi"]) for _ in range(count)]


def _inputs(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "solve3d":
        x, q, lb, ub = _points(case["dist"], case["n"], g)
        return dict(x=x, q=q, lb=lb, ub=ub)
    if kind == "forest3d":
        xs, qs, offs = [], [], [0]
        for i, n in enumerate(_sizes(case, case["systems"])):
            x, q, lb, ub = _points("uniform" if i % 2 == 0 else "blobs", n, g)
            xs.append(x)
            qs.append(q)
            offs.append(offs[-1] + n)
        return dict(x=torch.cat(xs), q=torch.cat(qs), lb=lb, ub=ub, offs=offs)
    if kind == "batch2d":
        offs = [0]
        for n in _sizes(case, case["systems"]):
            offs.append(offs[-1] + n)
        n = offs[-1]
        return dict(x=2 * _u(g, n, 2) - 1, q=2 * _u(g, n) - 1, offs=offs)
    sets = []
    for i, n in enumerate(_sizes(case, case["requests"])):
        x, q, _, _ = _points("plummer" if i % 2 else "uniform", n, g)
        sets.append(dict(x=x, q=q, tol=TOLERANCES[i % 3]))
    return dict(sets=sets)


_SERVED = dict(lbound=(-1.0, -1.0, -1.0), ubound=(1.0, 1.0, 1.0), maxbox=64, order=0, field=True)


def prepare(case, seed):
    inp = _inputs(case, seed)
    kind = case["kind"]
    st = dict(kind=kind, single=case.get("precision") == "mixed")
    if kind == "solve3d":
        st["solver"] = aran_gb300.Solver3d(
            inp["lb"], inp["ub"], maxbox=case["maxbox"], order=case["order"],
            flavour=case["flavour"], field=case["field"], precision=case["precision"])
        st["host"] = case["host"]
        if case["host"]:
            st["x"], st["q"] = inp["x"].cpu().numpy(), inp["q"].cpu().numpy()
        else:
            n = case["n"]
            st["x"], st["q"] = inp["x"], inp["q"]
            st["pot"] = torch.empty(n, device="cuda", dtype=torch.float64)
            st["fld"] = (torch.empty(n, 3, device="cuda", dtype=torch.float64) if case["field"]
                         else None)
    elif kind == "forest3d":
        st["solver"] = aran_gb300.Solver3d(inp["lb"], inp["ub"], maxbox=case["maxbox"],
                                           order=case["order"], field=case["field"],
                                           precision=case["precision"])
        st["x"], st["q"] = inp["x"].cpu().numpy(), inp["q"].cpu().numpy()
        st["offs"] = np.array(inp["offs"], np.int64)
        st["boxes"] = np.tile(np.array(inp["lb"] + inp["ub"]), (case["systems"], 1))
    elif kind == "batch2d":
        st["solver"] = aran_gb300.Solver2d(maxbox=case["maxbox"], order=case["order"],
                                           precision=case["precision"])
        st["x"], st["q"], st["offs"] = inp["x"], inp["q"], np.array(inp["offs"], np.int64)
        st["acc"] = torch.empty(len(inp["q"]), device="cuda", dtype=torch.complex128)
    else:
        # the loop as a service keeps it: its workers' solvers already exist
        st["server"] = aran_gb300.Server(nslots=case["slots"])
        st["sets"] = [dict(x=s["x"].cpu().numpy(), q=s["q"].cpu().numpy(), tol=s["tol"])
                      for s in inp["sets"]]
        st["single"] = [aran_gb300.plan_for_tolerance(s["tol"])[1] == "mixed" for s in st["sets"]]
        w = np.random.default_rng(0).uniform(0.0, 1.0, (4000, 3))
        for tol in TOLERANCES:
            tickets = [st["server"].submit(w, w[:, 0], tolerance=tol, **_SERVED)
                       for _ in range(3 * case["slots"])]
            for t in tickets:
                st["server"].wait(t)
    torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------- runs
def _out(single, pot, fld):
    if single:
        if isinstance(pot, np.ndarray):
            pot = pot.astype(np.float32)
            fld = None if fld is None else fld.astype(np.float32)
        else:
            pot = pot.float()
            fld = None if fld is None else fld.float()
    return {"pot": pot} if fld is None else {"pot": pot, "field": fld}


def run(st):
    kind = st["kind"]
    if kind == "solve3d":
        if st["host"]:
            return _out(st["single"], *st["solver"].solve(st["x"], st["q"]))
        fld = st["fld"]
        st["solver"].solve_device(len(st["q"]), st["x"].data_ptr(), st["q"].data_ptr(),
                                  st["pot"].data_ptr(), None if fld is None else fld.data_ptr())
        return _out(st["single"], st["pot"], fld)
    if kind == "forest3d":
        return _out(st["single"], *st["solver"].solve_forest(st["x"], st["q"], st["offs"],
                                                             st["boxes"]))
    if kind == "batch2d":
        st["solver"].solve_device(len(st["q"]), st["x"].data_ptr(), st["q"].data_ptr(),
                                  st["acc"].data_ptr(), st["offs"])
        return {"acc": st["acc"].to(torch.complex64) if st["single"] else st["acc"]}
    tickets = [st["server"].submit(s["x"], s["q"], tolerance=s["tol"], **_SERVED)
               for s in st["sets"]]
    outs = []
    for single, t in zip(st["single"], tickets):
        pot, fld, _ = st["server"].wait(t)
        outs.append(_out(single, pot, fld))
    return outs


# ------------------------------------------------------------------- exact
MOST_PAIRS = 9.1e10   # an FP64 direct sum of so many pairs stays within seconds


def _direct3d(x, q, field):
    """Newton potential and field by the FP64 direct sum; the field kernel
    leaves out pairs within 1e-5."""
    n = len(q)
    pot = torch.empty(n, device="cuda", dtype=torch.float64)
    fld = torch.empty(n, 3, device="cuda", dtype=torch.float64) if field else None
    xs = [x[:, k].contiguous() for k in range(3)]
    step = max(1, min(n, (1 << 26) // n))
    guard = 1e-10 if field else 0.0
    for a in range(0, n, step):
        b = min(n, a + step)
        d = [xs[k][a:b, None] - xs[k][None, :] for k in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        r2.masked_fill_(r2 <= guard, math.inf)
        inv = r2.rsqrt()
        w = inv * q
        pot[a:b] = w.sum(dim=1)
        if field:
            w.mul_(inv).mul_(inv)
            for k in range(3):
                fld[a:b, k] = -(d[k].mul_(w)).sum(dim=1)
    return pot, fld


def _direct2d(x, q):
    n = len(q)
    acc = torch.empty(n, 2, device="cuda", dtype=torch.float64)
    xs, ys = x[:, 0].contiguous(), x[:, 1].contiguous()
    step = max(1, min(n, (1 << 26) // n))
    for a in range(0, n, step):
        b = min(n, a + step)
        dx, dy = xs[a:b, None] - xs[None, :], ys[a:b, None] - ys[None, :]
        r2 = (dx * dx).addcmul_(dy, dy)
        r2.masked_fill_(r2 == 0, math.inf)
        w = q / r2
        acc[a:b, 0] = dx.mul_(w).sum(dim=1)
        acc[a:b, 1] = -dy.mul_(w).sum(dim=1)
    return torch.view_as_complex(acc)


def exact(case, seed):
    """The direct sums in FP64 (None where they would take too long)."""
    kind = case["kind"]
    if kind == "solve3d":
        if float(case["n"]) ** 2 > MOST_PAIRS:
            return None
        inp = _inputs(case, seed)
        return _out(False, *_direct3d(inp["x"], inp["q"], case["field"]))
    inp = _inputs(case, seed)
    if kind == "served":
        if sum(float(len(s["q"])) ** 2 for s in inp["sets"]) > MOST_PAIRS:
            return None
        return [_out(False, *_direct3d(s["x"], s["q"], True)) for s in inp["sets"]]
    spans = list(zip(inp["offs"], inp["offs"][1:]))
    if sum(float(b - a) ** 2 for a, b in spans) > MOST_PAIRS:
        return None
    if kind == "forest3d":
        outs = [_direct3d(inp["x"][a:b], inp["q"][a:b], case["field"]) for a, b in spans]
        return _out(False, torch.cat([o[0] for o in outs]),
                    torch.cat([o[1] for o in outs]) if case["field"] else None)
    return {"acc": torch.cat([_direct2d(inp["x"][a:b], inp["q"][a:b]) for a, b in spans])}


# -------------------------------------------------------------------- work
def _occupancy(dist, n, maxbox):
    """Points per leaf: cells of the octree's level for a uniform set, the
    mean of an adaptive tree otherwise."""
    if dist == "uniform":
        occ = float(n)
        while occ > maxbox:
            occ /= 8.0
        return max(1.0, occ)
    return max(1.0, min(n, 0.45 * maxbox))


def _work3d(dist, n, p, maxbox, field):
    """Algorithmic flops of one solve: pairs of neighbouring leaves, 189
    translations a node by the rotate operator's definition, the passes up
    and down, P2M and L2P; bytes: particles in, results out."""
    tri = lambda k: k * (k + 1) / 2                              # noqa: E731
    blk = lambda k: (k + 1) * (k + 2) * (4 * k + 3) / 6          # noqa: E731
    occ = _occupancy(dist, n, maxbox)
    nodes = 8.0 / 7.0 * n / occ
    m2l = 4 * (blk(p - 1) + p * (p + 1) * (p + 2) / 3 + blk(p))
    vert = 8 * blk(p - 1) + 8 * blk(p) + 8 * p * (p + 1) * (p + 2) / 6
    flops = n * min(27 * occ, n) * (20 if field else 11)
    flops += nodes * (min(189.0, nodes) * m2l + vert)
    flops += n * (16 * tri(p) + (32 if field else 12) * tri(p + 1))
    return {"bytes": float(n) * (32 + (32 if field else 8)), "flops": float(flops)}


def _mean_size(case):
    lo, hi = case["nlo"], case["nhi"]
    return lo if lo == hi else (hi - lo) / math.log(hi / lo)


def work(case):
    kind = case["kind"]
    if kind == "solve3d":
        return _work3d(case["dist"], case["n"], case["order"], case["maxbox"], case["field"])
    n = int(_mean_size(case))
    if kind == "forest3d":
        w = _work3d("blobs", n, case["order"], case["maxbox"], case["field"])
        return {k: v * case["systems"] for k, v in w.items()}
    if kind == "served":
        ws = [_work3d("blobs", n, p, 64, True) for p in (8, 16, 26)]
        return {k: sum(w[k] for w in ws) / 3 * case["requests"] for k in ("bytes", "flops")}
    p = case["order"]
    occ = 0.45 * case["maxbox"]
    nodes = 4.0 / 3.0 * n / occ
    flops = n * 9 * occ * 12 + nodes * 27 * 8 * (p + 1) * (p - 1) + n * 16 * p
    return {"bytes": 40.0 * n * case["systems"], "flops": flops * case["systems"]}
