"""Set-up of a batch: obstacle programs against the reference's loops replayed cell by cell
(update's pressure copy, Version-6-26-04.c:1153-1177; coefsc's additions, :939-963), cases that
share one program, inlet profiles that come and go, and a gradient's directions seeded and read
back together against the same directions one by one."""
import ctypes as C
import random

import numpy as np
import pytest

from conftest import assert_bitexact


class _Prog(C.Structure):
    _fields_ = [("ncopy", C.c_int), ("dst", C.POINTER(C.c_int)), ("src", C.POINTER(C.c_int)), ("hazard", C.c_int),
                ("nseq", C.c_int), ("cells", C.POINTER(C.c_int)), ("codes", C.POINTER(C.c_uint)),
                ("max_adds", C.c_int), ("touches_outlet", C.c_int), ("owners", C.POINTER(C.c_int)),
                ("fan", C.POINTER(C.c_int))]


def _replay(ranges, nx, ny):
    origin, seq = {}, {}
    for i0, i1, j0, j1 in ranges:
        copies = [((j0, i), (j0 - 1, i)) for i in range(i0, i1 + 1)] + [((j1, i), (j1 + 1, i)) for i in range(i0, i1 + 1)]
        copies += [((j, i0), (j, i0 - 1)) for j in range(j0, j1 + 1)] + [((j, i1), (j, i1 + 1)) for j in range(j0, j1 + 1)]
        for d, s in copies:
            origin[d] = origin.get(s, s)
        for i in range(i0, i1 + 1):
            for j in range(j0, j1 + 1):
                for t, (y, x) in enumerate(((j, i - 1), (j, i + 1), (j - 1, i), (j + 1, i))):
                    if 1 <= x <= nx - 2 and 1 <= y <= ny - 2:
                        seq.setdefault(y * nx + x, []).append(t)
    at = lambda c: c[0] * nx + c[1]
    return {at(d): at(s) for d, s in origin.items() if d != s}, seq


@pytest.mark.parametrize("seed", range(12))
def test_obstacle_programs(seed):
    import mgfvm
    from mgfvm import configs
    L = mgfvm.lib()
    rng = random.Random(seed)
    ng = 1 + seed % 3
    bx, by = rng.randint(4, 18), rng.randint(4, 18)
    obs = []
    for _ in range(rng.randint(1, 7)):
        a, c = rng.randint(1, bx), rng.randint(1, by)
        obs.append((a, min(bx, a + rng.randint(0, 3)), c, min(by, c + rng.randint(0, 3))))
    cfg = configs.small(32, ng, isolve=2, nfx=bx << (ng - 1), nfy=by << (ng - 1)).replace(ig_obs=ng, ibeg_obs=0, obstacles=obs)
    cc, keep = cfg.to_c()
    for ig in range(ng):
        nx, ny = (cfg.nfx >> ig) + 2, (cfg.nfy >> ig) + 2
        copies, seq = _replay(mgfvm.obstacle_ranges(cfg, ig), nx, ny)
        g = _Prog()
        rc = L.mgfvm_build_obstacle_prog(C.byref(cc), ig, C.byref(g))
        if max((len(v) for v in seq.values()), default=0) > 14:
            assert rc != 0
            continue
        assert rc == 0
        assert [(g.dst[k], g.src[k]) for k in range(g.ncopy)] == sorted(copies.items())
        code = {x: sum(t << (2 * k) for k, t in enumerate(v)) | len(v) << 28 for x, v in seq.items()}
        assert [(g.cells[k], g.codes[k]) for k in range(g.nseq)] == sorted(code.items())
        assert g.max_adds == max((len(v) for v in seq.values()), default=0)
        assert bool(g.hazard) == any(s in copies for s in copies.values())
        if g.fan:
            fan = [(g.fan[2 * k] & ~(1 << 30), g.fan[2 * k + 1]) for k in range(g.ncopy)]
            own = [g.owners[k] for k in range(g.ncopy)]
            assert own == sorted(own)
            assert {d: (o if s < 0 else s) for o, (d, s) in zip(own, fan)} == copies
            assert [bool(g.fan[2 * k] >> 30) for k in range(g.ncopy)] == [a != b for a, b in zip(own, own[1:] + [None])]
        else:
            assert g.hazard or g.ncopy == 0
        L.mgfvm_free_obstacle_prog(C.byref(g))


def _cfg(n, ngrid, obstacles, **kw):
    from mgfvm import configs
    return configs.small(32, ngrid, isolve=2, nfx=n, nfy=n, ig_obs=ngrid, obstacles=obstacles, **kw)


@pytest.mark.gpu
def test_shared_programs(oracle_built):
    from mgfvm import Solver
    from oracle import OracleCase
    A, B = [(3, 4, 2, 5), (8, 8, 7, 9)], [(5, 6, 9, 12)]
    cfgs = [_cfg(64, 3, o, amuf=1.0 / (20 + k)) for k, o in enumerate((A, A, B, B, [], [], A, A))]
    cfgs += [_cfg(64, 2, [(3, 4, 2, 5)]), _cfg(48, 2, [(3, 4, 2, 5)])]
    prof = [np.linspace(0.5, 1.5, 64), np.linspace(1.0, 2.0, 64), np.zeros(0), np.full(64, 0.7)]
    with Solver(cfgs) as s:
        for k, p in ((1, prof[0]), (6, prof[1]), (1, prof[2]), (3, prof[3])):   # (case 1's comes and goes)
            s.set_inlet_profile(k, p)
        s.cycle(3)
        for k, c in enumerate(cfgs):
            o = OracleCase(c, {6: prof[1], 3: prof[3]}.get(k))
            o.cycle(3)
            for f in ("u", "v", "p", "sc"):
                assert_bitexact(s.field(k, 0, f), o.get(0, f), f"case {k} {f}")
            o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nfx,nfy,ngrid", [(32, 24, 1), (16, 136, 3), (32, 32, 3)])   # (rows above and below a block's)
def test_gradient_directions(nfx, nfy, ngrid):
    import mgfvm
    from mgfvm import Solver, configs
    cfg = configs.small(32, ngrid, isolve=2, nfx=nfx, nfy=nfy, xl=nfx / nfy, yl=1.0)
    J, g, ga, gp = mgfvm.gradient(cfg, cycles=2)
    with Solver([cfg], tangent=True) as s:
        for kind, index, want in [("inlet", k, g[k]) for k in (0, 1, nfy // 2, nfy - 1)] + [("amuf", 0, ga), ("prsc", 0, gp)]:
            s.set_direction(0, kind, index)
            for ig in range(ngrid):
                t = s.tangent(0, ig, "u")
                col = np.zeros((nfy >> ig) + 2)
                if kind == "inlet":
                    col[(index >> ig) + 1] = 0.5 ** ig
                assert np.array_equal(t[:, 0], col) and not t[:, 1:].any()
            s.cycle(2)
            j, dj = s.objective(0)
            assert j == J and dj == want
