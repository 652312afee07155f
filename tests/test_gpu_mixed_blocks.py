"""Mixed precision's register-blocked smoother against the pair smoother (which a tuning of its
threads selects), bit for bit: one tile, a cell more, many tiles and
launches, odd launch counts, obstacles, cases of two sizes and cases that stop."""
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "p", "pp", "sc", "apu", "apv"]


def _cfg(nx, ny, ngrid, k=0, **kw):
    from mgfvm import configs
    w, h = nx >> (ngrid - 1), ny >> (ngrid - 1)
    return configs.small(32, ngrid, isolve=2, nfx=nx, nfy=ny, xl=nx / ny, yl=1.0, ig_obs=ngrid, sc_obs=0.2,
                         amuf=1.0 / (20.0 + 3 * k), obstacles=[(w // 4, w // 4 + w // 8, h // 3, h // 3 + h // 8)], **kw)


def _compare(cfgs, run):
    from mgfvm import Solver
    ng = max(c.ngrid for c in cfgs)
    with Solver(cfgs, precision="mixed") as a, Solver(cfgs, precision="mixed") as b:
        assert any(k == "smooth_mixed" for k, _, _ in a.profile_cycle())
        b.profile_cycle()
        b.set_tuning(smooth_threads=[1024] * ng)
        run(a)
        run(b)
        for k, c in enumerate(cfgs):
            for ig in range(c.ngrid):
                for f in STATE:
                    assert_bitexact(a.field(k, ig, f), b.field(k, ig, f), f"case {k} level {ig} {f}")


@pytest.mark.parametrize("nx,ny,ngrid,nswpm,nswpp", [
    (52, 54, 2, 2, 10),       # one region, whole
    (54, 56, 2, 2, 10),
    (102, 98, 2, 1, 3),
    (256, 128, 4, 2, 10),
    (300, 64, 3, 3, 7),
    (128, 400, 3, 5, 13),
])
@pytest.mark.parametrize("ncases", [1, 14])
def test_bitexact(nx, ny, ngrid, nswpm, nswpp, ncases):
    _compare([_cfg(nx, ny, ngrid, k, nswpm=nswpm, nswpp=nswpp) for k in range(ncases)], lambda s: s.cycle(3))


def test_sizes_and_stops():
    cfgs = [_cfg(*((128, 128, 3), (96, 160, 3))[k % 2], k, convergence=(1e30, 1e-30, 1e-30)[k % 3]) for k in range(9)]
    _compare(cfgs, lambda s: s.solve(5))
