"""The Gauss-Seidel smoother by a table of tiles (more tiles than SMs) against the oracle, bit
for bit: as many tiles as SMs and a few more, batches of several sizes (cases without a tile
where another has many), cases that stop while others go on, rows that are no multiple of 16
bytes (no table), and a wait for copies that runs out."""
import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "p", "pp", "sc", "su", "apu", "apv"]


def _cfg(nx, ny, ngrid, k=0, **kw):
    from mgfvm import configs
    w, h = nx >> (ngrid - 1), ny >> (ngrid - 1)
    return configs.small(32, ngrid, isolve=2, nfx=nx, nfy=ny, xl=nx / ny, yl=1.0, ig_obs=ngrid, sc_obs=0.2,
                         amuf=1.0 / (20.0 + 3 * k),
                         obstacles=[(w // 4, w // 4 + w // 8, h // 3, h // 3 + h // 8), (w // 2, w // 2, h // 2, h // 2 + 1)], **kw)


def _compare(cfgs, cycles, cases, band):
    from mgfvm import Solver
    from oracle import OracleCase
    with Solver(cfgs) as s:
        s.set_tuning(band_visit=[1] * band)
        s.cycle(cycles)
        for k in cases:
            o = OracleCase(cfgs[k])
            o.cycle(cycles)
            for ig in range(cfgs[k].ngrid):
                for f in STATE:
                    assert_bitexact(s.field(k, ig, f), o.get(ig, f), f"case {k} level {ig} {f}")
            o.close()


@pytest.mark.parametrize("nx,ny,ngrid,ncases", [
    (88, 92, 2, 37),      # 148 tiles of two by two at four and at five units
    (88, 92, 2, 38),
    (88, 92, 2, 75),      # two rounds and a tile
    (89, 92, 1, 60),      # an odd row
    (46, 48, 1, 160),     # a tile a case, every unit in one launch
    (400, 32, 2, 60),
    (32, 400, 2, 60),
])
def test_bitexact(nx, ny, ngrid, ncases, oracle_built):
    _compare([_cfg(nx, ny, ngrid, k) for k in range(ncases)], 3, (0, ncases // 2, ncases - 1), ngrid)


def test_wide_obstacle(oracle_built):
    """Values fall below the normal range deep inside (u, v by 1e-30 a cell, p' by 1e-60)."""
    from mgfvm import configs
    cfgs = [configs.small(32, 2, isolve=2, nfx=200, nfy=200, ig_obs=2, amuf=1.0 / (20.0 + k), obstacles=[(20, 80, 20, 80)])
            for k in range(10)]
    _compare(cfgs, 6, (0, 9), 2)


def test_sizes(oracle_built):
    cfgs = [_cfg(*((256, 128, 3), (64, 64, 2), (128, 200, 3))[k % 3], k) for k in range(30)]
    _compare(cfgs, 2, (0, 1, 2, 27, 28, 29), 3)


def test_cases_that_stop(oracle_built):
    """Every case of a solve with a stop test has the state and history of a solve of its own."""
    from mgfvm import Solver
    cfgs = [_cfg(96, 96, 3, k, convergence=(1e30, 1e-3, 1e-30)[k % 3]) for k in range(48)]
    with Solver(cfgs) as s:
        s.solve(12)
        for k in (0, 1, 2, 45, 46, 47):
            with Solver([cfgs[k]]) as one:
                one.solve(12)
                assert np.array_equal(s.history(k)[0], one.history(0)[0]) or np.allclose(
                    s.history(k)[0], one.history(0)[0], rtol=1e-12, atol=0)
                assert len(s.history(k)[0]) == len(one.history(0)[0])
                for f in STATE:
                    assert_bitexact(s.field(k, 0, f), one.field(0, 0, f), f"case {k} {f}")


def test_wait_runs_out():
    """Copies that are not waited for: the call fails, and after a reset the same cycles run."""
    from mgfvm import MgfvmError, Solver
    from mgfvm._abi import ETIMEOUT
    cfgs = [_cfg(128, 128, 3, k) for k in range(40)]
    with Solver(cfgs) as s, Solver(cfgs) as want:
        s.set_tuning(tma_first_wait=-1)
        with pytest.raises(MgfvmError) as ei:
            s.cycle(1)
        assert ei.value.status == ETIMEOUT
        s.set_tuning(tma_first_wait=0)
        s.reset()
        s.cycle(2)
        want.cycle(2)
        for f in STATE:
            assert_bitexact(s.field(39, 0, f), want.field(39, 0, f), f)
