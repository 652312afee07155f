"""Whole-level visits (a cluster of three CTAs a case) against the oracle, bit for bit: padded
levels on either side of the block size that leaves a thread its registers, odd rows, the
smallest level and the largest, both smoothers, odd sweep counts, periodic and fixed-pressure
sides, obstacles whose pressure copies chain, a batch of two sizes."""
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "p", "pp", "sc", "su", "apu", "apv"]


def _compare(cfgs, cycles):
    from mgfvm import Solver
    from oracle import OracleCase
    with Solver(cfgs) as s:
        kinds = {k for k, _, _ in s.profile_cycle()}
        assert "level_visit" in kinds
        s.cycle(cycles)
        for k, c in enumerate(cfgs):
            o = OracleCase(c)
            o.cycle(cycles + 1)
            for ig in range(c.ngrid):
                for f in STATE:
                    assert_bitexact(s.field(k, ig, f), o.get(ig, f), f"case {k} level {ig} {f}")
            o.close()


def _cfg(nx, ny, ngrid, isolve, **kw):
    from mgfvm import configs
    return configs.small(32, ngrid, isolve=isolve, nfx=nx, nfy=ny, xl=nx / ny, yl=1.0, **kw)


@pytest.mark.parametrize("isolve", [1, 2])
@pytest.mark.parametrize("nx,ny,ngrid,kw", [
    (34, 32, 1, {}),                          # 612 threads
    (34, 34, 1, {}),                          # 648
    (68, 68, 2, {}),                          # 648 on level 1, assembled by the restriction and by the visit
    (42, 42, 1, dict(nswpm=3, nswpp=7)),      # 968
    (31, 29, 1, dict(nswpm=1, nswpp=3)),      # odd rows
    (500, 2, 1, {}),                          # 1004, two rows
    (2, 500, 1, {}),
    (8, 8, 3, {}),                            # down to 2 x 2 cells
    (128, 64, 4, dict(ig_obs=4, sc_obs=0.2, obstacles=[(3, 4, 2, 3), (8, 9, 5, 6)])),
    (64, 64, 3, dict(ig_obs=3, sc_obs=0.2, obstacles=[(3, 4, 2, 3), (5, 6, 3, 4)])),   # touching: chained copies
])
def test_bitexact(isolve, nx, ny, ngrid, kw, oracle_built):
    _compare([_cfg(nx, ny, ngrid, isolve, **kw)], 2)


@pytest.mark.parametrize("isolve", [1, 2])
@pytest.mark.parametrize("sides", [dict(ibc_xm=3, ibc_xp=3), dict(ibc_ym=3, ibc_yp=3), dict(ibc_xm=2, ibc_xp=2),
                                   dict(ibc_ym=2, ibc_yp=2)])
def test_sides(isolve, sides, oracle_built):
    _compare([_cfg(48, 32, 3, isolve, **sides)], 2)


def test_two_sizes(oracle_built):
    _compare([_cfg(64, 72, 3, 2), _cfg(32, 24, 2, 2), _cfg(64, 72, 3, 2, amuf=0.02)], 2)
