"""The cycle that stops a case is done whole: after a solve that stops at once, every array
of every case is that of one V-cycle, also where the launch that ends the cycle has more
blocks than fit on the device at a time, and where the mass error is not finite."""
import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "p", "pp", "sc"]


def _compare(a, b, cases, levels):
    for k in cases:
        assert_bitexact(a.history(k)[0].view(np.int64), b.history(k)[0].view(np.int64), f"case {k} history")
        for ig in range(levels):
            for f in STATE:
                assert_bitexact(a.field(k, ig, f).view(np.int64), b.field(k, ig, f).view(np.int64), f"case {k} level {ig} {f}")


@pytest.mark.parametrize("n,ngrid,ncases,isolve", [(1024, 5, 1, 2), (1024, 1, 1, 2), (256, 4, 24, 2), (256, 4, 25, 1)])
def test_stops_at_once(n, ngrid, ncases, isolve):
    from mgfvm import Solver, configs
    cfgs = [configs.small(n, ngrid, isolve=isolve, nswpm=2, nswpp=4, amuf=1.0 / (20.0 + k), convergence=1e30)
            for k in range(ncases)]
    with Solver(cfgs) as s, Solver(cfgs) as want:
        want.cycle(1)
        for _ in range(3):
            s.reset()
            assert list(s.solve(9)) == [1] * ncases
            _compare(s, want, range(ncases), ngrid)


@pytest.mark.parametrize("n,ngrid", [(1024, 5), (512, 1)])
def test_not_finite(n, ngrid):
    from mgfvm import Solver, configs
    cfg = configs.small(n, ngrid, isolve=2)
    with Solver(cfg) as s, Solver(cfg) as want:
        for x in (s, want):
            u = x.field(0, 0, "u")
            u[n // 2, n // 2] = np.inf
            x.set_field(0, 0, "u", u)
        want.cycle(1)
        assert list(s.solve(9, allow_nonfinite=True)) == [1]
        _compare(s, want, [0], ngrid)


def test_others_go_on():
    """Cases that stop at once, later and never in one batch."""
    from mgfvm import Solver, configs
    cfgs = [configs.small(256, 4, isolve=2, nswpp=4, amuf=1.0 / (20.0 + k), convergence=(1e30, 1e-30)[k % 2]) for k in range(24)]
    with Solver(cfgs) as s, Solver(cfgs) as one, Solver(cfgs) as six:
        one.cycle(1)
        six.cycle(6)
        assert list(s.solve(6)) == [1, 6] * 12
        _compare(s, one, range(0, 24, 2), 1)
        _compare(s, six, range(1, 24, 2), 1)
