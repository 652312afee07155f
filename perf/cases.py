"""Workloads by which the engine's speed is followed, from a single small channel to
batches of obstacle flows, with the derivatives and the kernels a caller runs on its
own level storage.

`listed()` names them, `draw(rng)` gives another of the same ranges, `prepare` makes
what a program holds before the call (inputs, an open `Solver`, device arrays), `run`
is one pass through the public entry points, `work` counts what a pass cannot do
without, and `exact` gives the results in plain torch FP64: the V-cycle written here
on whole padded arrays, its gradients by torch's own reverse mode.

Kinds of pass:
  solve      reset a held Solver and run `cycles` V-cycles of every case of the batch
             with the stop rule; the level-0 fields and the cycle counts.  What a
             program does most: thousands of cycles on one context.
  sweep      build a context, give every case its inlet profile, solve, read the fields
             to the host, release the context: one point of a parameter study.
  adjoint    every case's gradient by reverse mode on a held Solver.
  gradient   one case's gradient by forward mode (mgfvm.gradient).
  relax      a level the caller stores itself: the mass residual, then `sweeps` of the
             smoother on p' (red-black Gauss-Seidel in place, or Jacobi with scratch).
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multigrid-fvm_b200"))

import mgfvm  # noqa: E402
from mgfvm import CaseConfig, Solver  # noqa: E402
from mgfvm._lib import check  # noqa: E402

JACOBI, GS = 1, 2
FIELDS = ("u", "v", "p", "sc")


def listed():
    return [
        # the plain channel at the smallest size users run: launch latency
        flow("channel_64", 64, 64, 3, 1, cycles=200, isolve=JACOBI, obstacles="none"),
        # the obstacle-flow pair (Re 10 and 100) of the benchmark, in FP64
        flow("obstacle_256_pair", 256, 256, 5, 2, cycles=60),
        # a design study: many obstacle cases in one context
        flow("obstacle_256_batch", 256, 256, 5, 64, cycles=10),
        # one large, finely resolved lattice (quarter-cell moves, obstacles three levels down)
        flow("lattice_1024", 1024, 1024, 7, 1, cycles=16, obstacles="quarter"),
        # cases of 64, 128 and 256 cells sharing their launches
        flow("sizes_batch", 256, 256, 5, 36, cycles=12, sizes=3),
        # the mixed-precision option on a middle-sized batch
        flow("mixed_256_batch", 256, 256, 5, 12, cycles=24, precision="mixed"),
        # a ragged, non-square duct with inlet and outlet ports and odd sweep counts
        flow("duct_ports", 304, 112, 5, 3, cycles=50, isolve=JACOBI, obstacles="none", ports=True, nswpm=3, nswpp=7),
        # a parameter study's inner call: build, solve, read back, release
        dict(flow("sweep_128", 128, 128, 4, 8, cycles=40), kind="sweep"),
        # gradients of a batch by reverse mode
        dict(flow("adjoint_128", 128, 128, 4, 6, cycles=6), kind="adjoint"),
        # one case's gradient by forward mode (66 directions)
        dict(flow("gradient_64", 64, 64, 3, 1, cycles=4), kind="gradient"),
        # a caller's own level: p' by red-black Gauss-Seidel on a large grid
        dict(name="relax_gs_1024", kind="relax", nx=1024, ny=1024, isolve=GS, sweeps=10),
        # and by Jacobi on a small ragged one: the smallest call
        dict(name="relax_jacobi_90", kind="relax", nx=90, ny=70, isolve=JACOBI, sweeps=4),
    ]


def flow(name, nx, ny, ngrid, ncases, cycles, isolve=GS, obstacles="full", precision="fp64", sizes=1, ports=False,
         nswpm=2, nswpp=10):
    return dict(name=name, kind="solve", nx=nx, ny=ny, ngrid=ngrid, ncases=ncases, cycles=cycles, isolve=isolve,
                obstacles=obstacles, precision=precision, sizes=sizes, ports=ports, nswpm=nswpm, nswpp=nswpp)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _levels(n):
    """Levels of an n-cell grid down to at least 16 cells (the obstacles' base lattice; the
    iteration is not stable on lattices whose coarse levels lack their obstacles)."""
    return int(math.log2(n / 16)) + 1


def draw(rng):
    kind = rng.choice(["solve"] * 8 + ["sweep", "adjoint", "gradient", "relax", "relax"])
    if kind == "relax":
        return dict(kind=kind, nx=_log_int(rng, 30, 1024), ny=_log_int(rng, 30, 1024),
                    isolve=rng.choice([JACOBI, GS]), sweeps=rng.randint(1, 12))
    isolve = rng.choice([JACOBI, GS, GS])
    if kind == "gradient":
        n, ngrid = 8 * rng.randint(4, 8), 3
        c = flow("", n, n, ngrid, 1, cycles=rng.randint(1, 4), isolve=isolve, obstacles=rng.choice(["none", "full"]))
    elif kind == "adjoint":
        n = rng.choice([64, 96, 128])
        c = flow("", n, n, _levels(n), rng.randint(1, 6), cycles=rng.randint(1, 6), isolve=isolve)
    elif kind == "sweep":
        n = rng.choice([64, 96, 128])
        c = flow("", n, n, _levels(n), rng.randint(1, 8), cycles=rng.randint(5, 40), isolve=isolve)
    else:
        form = rng.choice(["square", "square", "batch", "sizes", "duct", "large"])
        precision = rng.choice(["fp64", "fp64", "fp64", "mixed"])
        nswpm, nswpp = rng.choice([1, 2, 2, 3]), rng.choice([5, 7, 10, 10])
        kw = dict(isolve=isolve, precision=precision, nswpm=nswpm, nswpp=nswpp)
        if form == "square":
            n = 16 * rng.randint(4, 16)
            c = flow("", n, n, _levels(n), _log_int(rng, 1, 24), cycles=rng.randint(4, 24),
                     obstacles=rng.choice(["none", "full", "half"]), **kw)
        elif form == "batch":
            n = rng.choice([64, 128, 192, 256])
            c = flow("", n, n, _levels(n), rng.randint(24, 64), cycles=rng.randint(2, 8), **kw)
        elif form == "sizes":
            c = flow("", 256, 256, 5, rng.randint(6, 36), cycles=rng.randint(4, 12), sizes=3, **kw)
        elif form == "duct":
            c = flow("", 16 * rng.randint(4, 24), 16 * rng.randint(2, 10), 5, rng.randint(1, 6),
                     cycles=rng.randint(10, 50), obstacles="none", ports=True, **kw)
        else:
            n = 64 * rng.randint(6, 16)
            c = flow("", n, n, _levels(n), 1, cycles=rng.randint(4, 16), obstacles=rng.choice(["none", "full"]), **kw)
    del c["name"]
    c["kind"] = kind
    return c


# ------------------------------------------------------------------ inputs
def _lattice(n, ngrid, shift, rng):
    """Square blocks one base cell wide, one in every 3 x 3 base cells, each moved by up
    to a base cell in steps of a full, half or quarter one.  The base grid is the coarsest
    level of at least 16 cells; finer steps live on the level that many halvings below it.
    Blocks keep a gap (closed corners make the iteration diverge)."""
    base = max(lv for lv in range(ngrid) if lv == 0 or n >> lv >= 16)
    halvings = {"full": 0, "half": 1, "quarter": 2}[shift]
    m = 1 << halvings
    cells = n >> (base - halvings)
    blocks = []
    for j in range(m, cells - 2 * m, 3 * m):
        for i in range(2 * m, cells - 3 * m, 3 * m):
            a, b = i + int(rng.integers(m + 1)), j + int(rng.integers(m + 1))
            blocks.append((a + 1, a + m, b + 1, b + m))
    return dict(ig_obs=base - halvings + 1, obstacles=blocks)


def _cases(case, seed):
    """The batch's configurations and per-face inlet profiles (parabolic, perturbed)."""
    rng = np.random.default_rng([20, seed])
    cases, profiles = [], []
    for k in range(case["ncases"]):
        shrink = k % case["sizes"]
        nx, ny, ngrid = case["nx"] >> shrink, case["ny"] >> shrink, case["ngrid"] - shrink
        re = 10.0 if k % 2 == 0 and case["ncases"] > 1 else float(rng.uniform(40.0, 100.0))
        cfg = CaseConfig(nfx=nx, nfy=ny, ngrid=ngrid, nvcycle=2000, nswpm=case["nswpm"], nswpp=case["nswpp"],
                         isolve=case["isolve"], xl=nx / ny, yl=1.0, amuf=1.0 / re, prsc=float(rng.uniform(0.7, 1.3)),
                         relxm=0.7, relxp=0.3, guess=(0.0, 0.0, 0.0, 0.3), sc_obs=0.2)
        if case["obstacles"] != "none":
            shift = case["obstacles"]
            cfg = cfg.replace(**_lattice(min(nx, ny), ngrid, case["obstacles"], rng))
        if case["ports"]:
            lv = ngrid - 1
            m = ny >> lv
            a = 1 + int(rng.integers(max(1, m // 2)))
            cfg = cfg.replace(ig_inlt=lv + 1, ig_outlt=lv + 1, bc_xm=(0.0, 0.0, 0.0, 0.0),
                              inlets=[(a, min(a + 1, m), float(rng.uniform(0.5, 1.0)), 0.0, 1.0)],
                              outlets=[(1, m, 0.1, 0.0, 0.0)])
        cases.append(cfg)
        profiles.append(1.0 + 0.1 * rng.standard_normal(ny))
    return cases, profiles


def _by_size(cases):
    """Indices of the cases of each grid size."""
    groups = {}
    for k, c in enumerate(cases):
        groups.setdefault((c.nfx, c.nfy), []).append(k)
    return list(groups.values())


def _level(case, seed):
    """A caller's own level on the device: face velocities and areas, p' coefficients of
    a fluid with solid cells (the diagonal's 1e30), zero p'."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(7919 * seed + 13)
    shape = (case["ny"] + 2, case["nx"] + 2)
    rnd = lambda lo, hi: lo + (hi - lo) * torch.rand(shape, generator=g, device=dev, dtype=torch.float64)
    t = dict(u=rnd(-1.0, 1.0), v=rnd(-1.0, 1.0), ax=torch.full(shape, 1.0 / case["ny"], dtype=torch.float64, device=dev),
             ay=torch.full(shape, 1.0 / case["nx"], dtype=torch.float64, device=dev))
    for k in ("aw", "ae", "as", "an"):
        t[k] = rnd(0.5, 1.5)
    t["ap"] = t["aw"] + t["ae"] + t["as"] + t["an"] + 1.0e30 * (rnd(0.0, 1.0) < 0.2)
    for k in ("su", "pp", "scratch"):
        t[k] = torch.zeros(shape, dtype=torch.float64, device=dev)
    return t


def prepare(case, seed):
    if case["kind"] == "relax":
        npx, npy = case["nx"] + 2, case["ny"] + 2
        t = _level(case, seed)
        n = mgfvm.lib().mgfvm_masserror_scratch_doubles(npx, npy)
        t["partials"] = torch.zeros(n, dtype=torch.float64, device="cuda")
        t["err"] = torch.zeros(1, dtype=torch.float64, device="cuda")
        return dict(case=case, t=t)
    cases, profiles = _cases(case, seed)
    st = dict(case=case, cases=cases, profiles=profiles)
    if case["kind"] in ("solve", "adjoint"):
        s = Solver(cases, precision=case["precision"])
        for k, pr in enumerate(profiles):
            if not case["ports"]:
                s.set_inlet_profile(k, pr)
        st["solver"] = s
        if case["kind"] == "solve":
            st["views"] = {f: [[s.field_view(k, 0, f) for k in idx] for idx in _by_size(cases)] for f in FIELDS}
            st["stream"] = torch.cuda.ExternalStream(s.stream)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        s = st["solver"]
        s.reset()
        ran = s.solve(case["cycles"])
        fields = {f: [torch.stack(g) for g in groups] for f, groups in st["views"].items()}
        st["stream"].wait_stream(torch.cuda.current_stream())   # the next pass writes what this one reads
        return dict(ran=ran, fields=fields)
    if kind == "sweep":
        with Solver(st["cases"], precision=case["precision"]) as s:
            for k, pr in enumerate(st["profiles"]):
                s.set_inlet_profile(k, pr)
            ran = s.solve(case["cycles"])
            fields = [{f: s.field(k, 0, f) for f in FIELDS} for k in range(len(st["cases"]))]
        return dict(ran=ran, fields=fields)
    if kind == "adjoint":
        s = st["solver"]
        s.adjoint(case["cycles"])
        return [s.adjoint_gradient(k) for k in range(len(st["cases"]))]
    if kind == "gradient":
        return [mgfvm.gradient(st["cases"][0], st["profiles"][0], cycles=case["cycles"])]
    t, L = st["t"], mgfvm.lib()
    npx, npy = case["nx"] + 2, case["ny"] + 2
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = {k: C.c_void_p(a.data_ptr()) for k, a in t.items()}
    check(L.mgfvm_masserror_f64(p["u"], p["v"], p["ax"], p["ay"], p["su"], p["pp"], npx, npy, p["err"],
                                p["partials"], stream))
    co = (p["aw"], p["ae"], p["as"], p["an"], p["ap"], p["su"])
    if case["isolve"] == GS:
        check(L.mgfvm_rbgs_f64(*co, p["pp"], npx, npy, npx - 1, npy - 1, case["sweeps"], stream))
    else:
        check(L.mgfvm_jacobi_f64(*co, p["pp"], p["scratch"], npx, npy, npx - 1, npy - 1, case["sweeps"], stream))
    return dict(pp=t["pp"], su=t["su"], err=t["err"])


# -------------------------------------------------------------------- work
def work(case):
    """Level-0 state in and out once and the arithmetic of the cycles: 11 operations a
    cell update of the smoothers, 110 a cell for a visit's assemblies, mass residual and
    update, 160 a fine cell for a transfer down and up (about 3 and 7 times as much for
    forward and reverse derivatives)."""
    if case["kind"] == "relax":
        n = case["nx"] * case["ny"]
        return dict(bytes=8.0 * 11 * n, flops=(11.0 * case["sweeps"] + 9.0) * n)
    cells = flops = 0.0
    for shrink in range(case["sizes"]):
        nx, ny, ngrid = case["nx"] >> shrink, case["ny"] >> shrink, case["ngrid"] - shrink
        share = case["ncases"] / case["sizes"]
        cells += share * nx * ny
        for ig in range(ngrid):
            n = share * (nx >> ig) * (ny >> ig)
            visits = 1 if ig in (0, ngrid - 1) else 2
            flops += n * (visits * (11.0 * (3 * case["nswpm"] + case["nswpp"]) + 110.0)
                          + (160.0 if ig < ngrid - 1 else 0.0))
    flops *= case["cycles"]
    if case["kind"] == "gradient":
        flops *= 3.0 * (case["ny"] + 2)
    elif case["kind"] == "adjoint":
        flops *= 7.0
    return dict(bytes=8.0 * 8 * cells, flops=flops)


# ------------------------------------------------- the same in plain FP64 torch
def exact(case, seed):
    if case["kind"] == "relax":
        return _exact_relax(case, seed)
    cases, profiles = _cases(case, seed)
    if case["ports"]:
        profiles = [None] * len(cases)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    out = [None] * len(cases)
    for idx in _by_size(cases):
        grad = case["kind"] in ("adjoint", "gradient")
        th = _theta([cases[k] for k in idx], [profiles[k] for k in idx], dev, grad)
        with torch.set_grad_enabled(grad):
            F = _Flow([cases[k] for k in idx], th, dev)
            for _ in range(case["cycles"]):
                F.cycle()
            a = F.x[0]
            if grad:
                p, sc, ny = a["p"], a["sc"], F.lv[0].ny - 2
                J = (p[:, 1:-1, 1].sum(1) / ny - p[:, 1:-1, -2].sum(1) / ny) + sc[:, 1:-1, -1].sum(1) / ny
                J.sum().backward()
        for b, k in enumerate(idx):
            if grad:
                g = [th[n].grad[b].cpu().numpy() for n in ("inlet", "amuf", "prsc")]
                out[k] = (float(J[b].detach()), g[0], float(g[1]), float(g[2]))
            else:
                out[k] = {f: a[f][b] for f in FIELDS}
    if case["kind"] in ("adjoint", "gradient"):
        return out
    if case["kind"] == "solve":
        out = {f: [torch.stack([out[k][f] for k in idx]) for idx in _by_size(cases)] for f in FIELDS}
    return dict(ran=None, fields=out)


def _exact_relax(case, seed):
    t = _level(case, seed)
    ax, ay, u, v = (t[k] for k in ("ax", "ay", "u", "v"))
    c, w, e = (slice(1, -1), slice(1, -1)), (slice(1, -1), slice(0, -2)), (slice(1, -1), slice(2, None))
    s, n = (slice(0, -2), slice(1, -1)), (slice(2, None), slice(1, -1))
    div = ax[c] * u[c] - ax[c] * u[w] + ay[c] * v[c] - ay[c] * v[s]
    su, pp = t["su"], t["pp"]
    su[c] = -div
    i, j = torch.arange(su.shape[1], device=su.device), torch.arange(su.shape[0], device=su.device)
    red = ((i[None, :] + j[:, None]) % 2 == 0)[c]
    for _ in range(case["sweeps"]):
        for colour in ((red, ~red) if case["isolve"] == GS else (None,)):
            nb = t["aw"][c] * pp[w] + t["ae"][c] * pp[e] + t["as"][c] * pp[s] + t["an"][c] * pp[n]
            if colour is None:
                pp[c] = (nb + su[c]) / (t["ap"][c] + 1.0e-30)
            else:
                pp[c] = torch.where(colour, (nb + su[c]) / t["ap"][c], pp[c])
    return dict(pp=pp, su=su, err=div.abs().sum().reshape(1))


def _theta(cases, profiles, dev, grad):
    """Inlet profiles, viscosities and Prandtl-type numbers of a group of cases."""
    th = dict(amuf=[c.amuf for c in cases], prsc=[c.prsc for c in cases])
    th = {k: torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=grad) for k, v in th.items()}
    th["inlet"] = None
    if profiles[0] is not None:
        th["inlet"] = torch.tensor(np.stack(profiles), dtype=torch.float64, device=dev, requires_grad=grad)
    return th


def _put(a, at, value):
    b = a.clone()
    b[at] = value
    return b


class _Lv:
    pass


class _Flow:
    """SIMPLE in FAS V-cycles on padded arrays (batch, y, x), every routine functional so
    torch can differentiate it: cases of one size with inflow at x-, walls at y-, y+ and
    outflow at x+ (or ports)."""

    def __init__(self, cases, th, dev):
        self.c0, self.B = cases[0], len(cases)
        col = lambda v: v.reshape(-1, 1, 1)
        self.amu, self.prsc = col(th["amuf"]), col(th["prsc"])
        self.amusc = self.amu / self.prsc
        self.rm, self.rp = self.c0.relxm, self.c0.relxp
        self.lv, self.x = [], []
        for ig in range(self.c0.ngrid):
            self._level(cases, ig, dev)
        if th["inlet"] is not None:
            u = self.x[0]["u"]
            self.x[0]["u"] = _put(u, (slice(None), slice(1, -1), 0), th["inlet"])
        for ig in range(1, self.c0.ngrid):
            for i in (0, -2):
                f, k = self.x[ig - 1], self.x[ig]
                for q in "uv":
                    a = f[q][:, :, 2 * (self.lv[ig].nx - 2) if i else 0]
                    if q == "u":
                        m = 0.5 * (a[:, 2:-1:2] + a[:, 1:-2:2])
                    else:
                        flat = f[q].reshape(self.B, -1)
                        at = torch.arange(2, self.lv[ig - 1].ny - 1, 2, device=dev) * self.lv[ig - 1].nx \
                            + (2 * (self.lv[ig].nx - 2) if i else 0)
                        m = 0.5 * (flat[:, at] + flat[:, at - 1])
                    k[q] = _put(k[q], (slice(None), slice(1, -1), i), m)

    def _level(self, cases, ig, dev):
        c = self.c0
        L = _Lv()
        L.nx, L.ny = c.nfx // (1 << ig) + 2, c.nfy // (1 << ig) + 2
        L.dx, L.dy = c.xl / (L.nx - 2), c.yl / (L.ny - 2)
        shape = (self.B, L.ny, L.nx)
        full = lambda v: torch.full(shape, float(v), dtype=torch.float64, device=dev)
        L.ax, L.ay = full(L.dy), full(L.dx)
        if ig:
            F = self.lv[ig - 1]
            L.ax[:, 1:-1, :-1] = F.ax[:, 2:-1:2, 0:-1:2] + F.ax[:, 1:-2:2, 0:-1:2]
            L.ay[:, :-1, 1:-1] = F.ay[:, 0:-1:2, 2:-1:2] + F.ay[:, 0:-1:2, 1:-2:2]
        x = dict(zip(("u", "v", "p", "sc"), (full(g) for g in c.guess)))
        for k in ("pp", "resu", "resv", "ressc"):
            x[k] = full(0.0)
        x["apu"], x["apv"] = full(1.0e30), full(1.0e30)
        every = slice(None)
        for side, at, bc in (("xm", (every, every, 0), c.bc_xm), ("xp", (every, every, -1), c.bc_xp),
                             ("ym", (every, 0), c.bc_ym), ("yp", (every, -1), c.bc_yp)):
            for q, val in zip(("u", "v", "p", "sc"), bc):
                x[q][(every, every, -2) if (q, side) == ("u", "xp") else at] = val
        L.spu, L.spv, L.spsc, L.solid = full(0.0), full(0.0), full(0.0), full(0.0)
        add = [full(0.0) for _ in range(4)]          # obstacle faces of the scalar: ae, aw, an, as
        copy = np.tile(np.arange(L.nx * L.ny), (self.B, 1))
        for b, cb in enumerate(cases):
            P = copy[b].reshape(L.ny, L.nx)
            for i0, i1, j0, j1 in mgfvm.obstacle_ranges(cb, ig):
                if i1 < i0 or j1 < j0:
                    continue
                J, I = slice(j0, j1 + 1), slice(i0, i1 + 1)
                W, S = slice(i0 - 1, i1), slice(j0 - 1, j1)
                E, N = slice(i0 + 1, i1 + 2), slice(j0 + 1, j1 + 2)
                for q in "uv":
                    x[q][b, J, I] = 0.0
                x["u"][b, J, W] = 0.0
                x["v"][b, S, I] = 0.0
                for a, r, s in ((L.spu, J, I), (L.spu, J, W), (L.spv, J, I), (L.spv, S, I), (L.spsc, J, I)):
                    a[b, r, s] = 1.0e30
                L.solid[b, J, I] = 1.0e30
                x["sc"][b, J, I] = cb.sc_obs
                add[0][b, J, W] += L.ax[b, J, I] / L.dx
                add[1][b, J, E] += L.ax[b, J, I] / L.dx
                add[2][b, S, I] += L.ay[b, J, I] / L.dy
                add[3][b, N, I] += L.ay[b, J, I] / L.dy
                P[j0, I] = P[j0 - 1, I]
                P[j1, I] = P[j1 + 1, I]
                P[J, i0] = P[J, i0 - 1]
                P[J, i1] = P[J, i1 + 1]
            for ports, igp, i in ((cb.inlets, cb.ig_inlt, 0), (cb.outlets, cb.ig_outlt, -2)):
                if ig >= igp:
                    continue
                m = 1 << (igp - 1 - ig)
                for jf, jl, u, v, sc in ports:
                    r = slice((jf - 1) * m + 1, jl * m + 1)
                    x["u"][b, r, i], x["v"][b, r, i], x["sc"][b, r, i + 1 if i else 0] = u, v, sc
        L.add = [a[:, 1:-1, 1:-1] for a in add]
        L.copy = torch.from_numpy(copy).to(dev)
        j, i = torch.arange(L.ny, device=dev)[:, None], torch.arange(L.nx, device=dev)[None, :]
        L.red = (i + j) % 2 == 0
        self.lv.append(L)
        self.x.append(x)

    # hybrid coefficients of u, v and the scalar on their domains
    @staticmethod
    def _hyb(c, d, sign):
        m = torch.maximum(c.abs(), d)
        return m + c if sign > 0 else m - c

    def _coef(self, ig, e):
        L, x = self.lv[ig], self.x[ig]
        cx, cy = 0.5 * x["u"] * L.ax, 0.5 * x["v"] * L.ay
        h = self._hyb
        if e == "u":
            c = (slice(None), slice(1, -1), slice(1, -2))
            cxm = 0.5 * (cx[c] + cx[:, 1:-1, 0:-3])
            cxp = 0.5 * (cx[c] + cx[:, 1:-1, 2:-1])
            cym = 0.5 * (cy[:, 0:-2, 1:-2] + cy[:, 0:-2, 2:-1])
            cyp = 0.5 * (cy[c] + cy[:, 1:-1, 2:-1])
            dx, dy = self.amu * (L.ax[c] / L.dx), self.amu * (L.ay[c] / L.dy)
        elif e == "v":
            c = (slice(None), slice(1, -2), slice(1, -1))
            cxm = 0.5 * (cx[:, 1:-2, 0:-2] + cx[:, 2:-1, 0:-2])
            cxp = 0.5 * (cx[c] + cx[:, 2:-1, 1:-1])
            cym = 0.5 * (cy[c] + cy[:, 0:-3, 1:-1])
            cyp = 0.5 * (cy[c] + cy[:, 2:-1, 1:-1])
            dx, dy = self.amu * (L.ax[c] / L.dx), self.amu * (L.ay[c] / L.dy)
        else:
            c = (slice(None), slice(1, -1), slice(1, -1))
            aw = h(cx[:, 1:-1, 0:-2], self.amusc * (L.ax[:, 1:-1, 0:-2] / L.dx), 1)
            ae = h(cx[c], self.amusc * (L.ax[c] / L.dx), -1)
            as_ = h(cy[:, 0:-2, 1:-1], self.amusc * (L.ay[:, 0:-2, 1:-1] / L.dy), 1)
            an = h(cy[c], self.amusc * (L.ay[c] / L.dy), -1)
            ap = aw + ae + as_ + an
            face = [self.amusc * a for a in L.add]
            ap = ap + (face[0] + face[1] + face[2] + face[3])
            return c, aw + face[1], ae + face[0], as_ + face[3], an + face[2], ap
        aw, ae, as_, an = h(cxm, dx, 1), h(cxp, dx, -1), h(cym, dy, 1), h(cyp, dy, -1)
        ap = aw + ae + as_ + an
        z = torch.zeros_like(ap)
        if e == "u":       # wall shear: top row, then bottom row (face area of the top row)
            a = self.amu * (L.ay[:, -2:-1, 1:-2] / L.dy)
            top, bot = _put(z, (slice(None), slice(-1, None)), a), _put(z, (slice(None), slice(0, 1)), a)
            return c, aw, ae, as_ + bot, an + top, ap + top + bot
        a = self.amu * (L.ay[:, 1:-2, -2:-1] / L.dy)
        rgt = _put(z, (slice(None), slice(None), slice(-1, None)), a)
        lft = _put(z, (slice(None), slice(None), slice(0, 1)), a)
        return c, aw + lft, ae + rgt, as_, an, ap + rgt + lft

    @staticmethod
    def _around(a, c):
        b, r, s = c
        sh = lambda t, k, n: slice(t.start + k, n + (t.stop + k))
        ny, nx = a.shape[1], a.shape[2]
        return (a[b, r, sh(s, -1, nx)], a[b, r, sh(s, 1, nx)], a[b, sh(r, -1, ny), s], a[b, sh(r, 1, ny), s])

    def _smooth(self, ig, field, co, su, sweeps):
        c, aw, ae, as_, an, ap = co
        L, x = self.lv[ig], self.x[ig]
        phi = x[field]
        red = L.red[c[1], c[2]]
        jac = self.c0.isolve == JACOBI
        for _ in range(sweeps):
            for colour in ((None,) if jac else (red, ~red)):
                w, e, s, n = self._around(phi, c)
                val = (aw * w + ae * e + as_ * s + an * n + su) / (ap + 1.0e-30 if jac else ap)
                phi = _put(phi, c, val if jac else torch.where(colour, val, phi[c]))
        x[field] = phi

    def _momentum(self, ig, q):
        L, x = self.lv[ig], self.x[ig]
        c, aw, ae, as_, an, ap = self._coef(ig, q)
        area, sp = (L.ax, L.spu) if q == "u" else (L.ay, L.spv)
        _, pe, _, pn = self._around(x["p"], c)
        ap = ap / self.rm
        su = area[c] * (x["p"][c] - (pe if q == "u" else pn)) + (1.0 - self.rm) * ap * x[q][c] + x["res" + q][c]
        ap = ap + sp[c]
        return (c, aw, ae, as_, an, ap), su

    def _outflow(self, ig, fields):
        if self.c0.ibc_xp != 4:
            return
        x, all_ = self.x[ig], slice(None)
        for f in fields:
            i = -2 if f == "u" else -1
            x[f] = _put(x[f], (all_, all_, i), x[f][:, :, i - 1])

    def _visit(self, ig, down):
        """fluxes, the three transport equations (each from the fluxes at the start), p'."""
        L, x, c0 = self.lv[ig], self.x[ig], self.c0
        co_u, su_u = self._momentum(ig, "u")
        co_v, su_v = self._momentum(ig, "v")
        k = list(self._coef(ig, "sc"))
        c = k[0]
        su_s = L.spsc[c] * c0.sc_obs + x["ressc"][c]
        k[5] = k[5] + L.spsc[c]
        self._smooth(ig, "u", co_u, su_u, c0.nswpm)
        self._smooth(ig, "v", co_v, su_v, c0.nswpm)
        x["apu"] = _put(x["apu"], co_u[0], co_u[5])
        x["apv"] = _put(x["apv"], co_v[0], co_v[5])
        u, v, ax, ay = x["u"], x["v"], L.ax, L.ay
        su = -(ax[c] * u[c] - ax[c] * u[:, 1:-1, :-2] + ay[c] * v[c] - ay[c] * v[:, :-2, 1:-1])
        aw, ae = ax[:, 1:-1, :-2] ** 2 / x["apu"][:, 1:-1, :-2], ax[c] ** 2 / x["apu"][c]
        as_, an = ay[:, :-2, 1:-1] ** 2 / x["apv"][:, :-2, 1:-1], ay[c] ** 2 / x["apv"][c]
        x["pp"] = _put(x["pp"], c, 0.0)
        self._smooth(ig, "pp", (c, aw, ae, as_, an, aw + ae + as_ + an + L.solid[c]), su, c0.nswpp)
        pp = x["pp"]
        x["u"] = _put(u, c, u[c] + ax[c] * (pp[c] - pp[:, 1:-1, 2:]) / x["apu"][c])
        x["v"] = _put(v, c, v[c] + ay[c] * (pp[c] - pp[:, 2:, 1:-1]) / x["apv"][c])
        p = _put(x["p"], c, x["p"][c] + self.rp * pp[c])
        x["p"] = torch.gather(p.reshape(self.B, -1), 1, L.copy).reshape(p.shape)
        if down:
            self._outflow(ig, ("u", "v", "p", "sc"))
            self._smooth(ig, "sc", k, su_s, c0.nswpm)
        else:
            self._smooth(ig, "sc", k, su_s, c0.nswpm)
            self._outflow(ig, ("u", "v", "p", "sc"))

    @staticmethod
    def _four(a):
        return a[:, 2:-1:2, 2:-1:2], a[:, 2:-1:2, 1:-2:2], a[:, 1:-2:2, 2:-1:2], a[:, 1:-2:2, 1:-2:2]

    def _restricted(self, ig):
        """Fine u, v, p, sc averaged onto the interior of level ig + 1."""
        F, K, x = self.lv[ig], self.lv[ig + 1], self.x[ig]
        c = (slice(None), slice(1, -1), slice(1, -1))
        u, _, us, _ = self._four(x["u"] * F.ax)
        v, vw, _, _ = self._four(x["v"] * F.ay)
        out = dict(u=(u + us) / (K.ax[c] + 1.0e-30), v=(v + vw) / (K.ay[c] + 1.0e-30))
        for f in ("p", "sc"):
            a, b, d, e = self._four(x[f])
            out[f] = 0.25 * (a + b + d + e)
        return out

    def _residual(self, ig, q, fine):
        L, x = self.lv[ig], self.x[ig]
        co = self._coef(ig, q)
        c, aw, ae, as_, an, ap = co
        w, e, s, n = self._around(x[q], c)
        r = aw * w + ae * e + as_ * s + an * n - ap * x[q][c]
        if q != "sc":
            area = L.ax if q == "u" else L.ay
            _, pe, _, pn = self._around(x["p"], c)
            r = r + area[c] * (x["p"][c] - (pe if q == "u" else pn))
        if fine:
            r = r + x["res" + q][c]
        return c, _put(torch.zeros_like(x[q]), c, r)

    def _restrict(self, ig):
        c = (slice(None), slice(1, -1), slice(1, -1))
        K = self.x[ig + 1]
        for f, a in self._restricted(ig).items():
            K[f] = _put(K[f], c, a)
        for q in ("u", "v", "sc"):
            _, r = self._residual(ig, q, True)
            ck, rc = self._residual(ig + 1, q, False)
            a, w, s, sw = self._four(r)
            if q == "u":
                e, se = r[:, 2:-1:2, 3::2], r[:, 1:-2:2, 3::2]
                d = (a + s) + 0.5 * (w + sw + e + se)
            elif q == "v":
                n, nw = r[:, 3::2, 2:-1:2], r[:, 3::2, 1:-2:2]
                d = (a + w) + 0.5 * (s + sw + n + nw)
            else:
                d = a + s + w + sw
            d = _put(torch.zeros_like(rc), c, d)
            K["res" + q] = _put(K["res" + q], ck, d[ck] - rc[ck])

    def _prolong(self, ig):
        F, fx, K, kx = self.lv[ig], self.x[ig], self.lv[ig + 1], self.x[ig + 1]
        c = (slice(None), slice(1, -1), slice(1, -1))
        R = self._restricted(ig)
        up, vp = self._four(F.spu)[0] > 1.0e10, self._four(F.spv)[0] > 1.0e10
        cc = {f: _put(torch.zeros_like(kx[f]), c, kx[f][c] - R[f]) for f in ("u", "v", "p", "sc")}
        cc["p"] = _put(cc["p"], c, torch.where(up, torch.zeros_like(cc["p"][c]), cc["p"][c]))
        rows, cols = slice(2, -1, 2), slice(1, -2, 2)
        # u: faces ic = 1 .. nxc-3, the rows above and below; v likewise
        m = cc["u"].clone()
        m[:, :, -2] = 0.0
        z = torch.zeros_like(m[c])
        c1 = torch.where(up, z, 0.75 * m[c] + 0.25 * m[:, 2:, 1:-1])[:, :, :-1]
        c2 = torch.where(up, z, 0.75 * m[c] + 0.25 * m[:, :-2, 1:-1])[:, :, :-1]
        u = fx["u"].clone()
        for r, d in ((rows, c1), (cols, c2)):
            u[:, r, 2:-3:2] = u[:, r, 2:-3:2] + d
            u[:, r, 3:-2:2] = u[:, r, 3:-2:2] + 0.5 * d
            u[:, r, 1:-4:2] = u[:, r, 1:-4:2] + 0.5 * d
        m = cc["v"].clone()
        m[:, -2] = 0.0
        c1 = torch.where(vp, z, 0.75 * m[c] + 0.25 * m[:, 1:-1, 2:])[:, :-1]
        c2 = torch.where(vp, z, 0.75 * m[c] + 0.25 * m[:, 1:-1, :-2])[:, :-1]
        v = fx["v"].clone()
        for s, d in ((rows, c1), (cols, c2)):
            v[:, 2:-3:2, s] = v[:, 2:-3:2, s] + d
            v[:, 3:-2:2, s] = v[:, 3:-2:2, s] + 0.5 * d
            v[:, 1:-4:2, s] = v[:, 1:-4:2, s] + 0.5 * d
        new = dict(u=u, v=v)
        for f in ("p", "sc"):
            a, m = fx[f].clone(), cc[f]
            for r, dj in ((rows, 1), (cols, -1)):
                for s, di in ((rows, 1), (cols, -1)):
                    j, i = slice(1 + dj, m.shape[1] - 1 + dj), slice(1 + di, m.shape[2] - 1 + di)
                    a[:, r, s] = a[:, r, s] + (9. / 16. * m[c] + 3. / 16. * m[:, 1:-1, i] + 3. / 16. * m[:, j, 1:-1]
                                               + 1. / 16. * m[:, j, i])
            new[f] = a
        fx.update(new)

    def cycle(self):
        ng = len(self.lv)
        for ig in range(ng):
            self._visit(ig, True)
            if ig != ng - 1:
                self._restrict(ig)
        for ig in range(ng - 1, 0, -1):
            self._prolong(ig - 1)
            if ig != 1:
                self._visit(ig - 1, False)
