"""The register-blocked Gauss-Seidel smoother (blocks of 2 x 4 cells, 54 x 56 regions) against
the oracle, bit for bit: odd and even row lengths (scalar and paired loads), domains one
cell around whole tiles, one tile, one launch and several, odd launch counts, one to twenty
units, obstacles (dividends far outside the plain range of the division) and a batch of two
sizes.  The batches are large enough that the schedule takes this smoother on level 0, which
the launch list confirms."""
import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "p", "pp", "sc", "su", "apu", "apv"]


def _cfg(nx, ny, ngrid, nswpm, nswpp, obstacles):
    from mgfvm import configs
    cfg = configs.small(32, ngrid, isolve=2, nfx=nx, nfy=ny, xl=nx / ny, yl=1.0, nswpm=nswpm, nswpp=nswpp)
    if obstacles:
        w, h = nx >> (ngrid - 1), ny >> (ngrid - 1)
        cfg = cfg.replace(ig_obs=ngrid, sc_obs=0.2,
                          obstacles=[(w // 4, w // 4 + w // 8, h // 3, h // 3 + h // 8), (w // 2, w // 2, h // 2, h // 2 + 1)])
    return cfg


@pytest.mark.parametrize("nx,ny,ngrid,nswpm,nswpp,ncases", [
    (201, 97, 1, 2, 10, 40),      # odd row length
    (132, 138, 2, 2, 10, 48),     # 44 x 46: whole tiles at four units
    (134, 140, 2, 1, 3, 48),      # a cell more; two and six units
    (90, 94, 1, 3, 7, 64),        # six units of u, v, sc; fourteen of p'
    (64, 64, 3, 2, 10, 5),        # one launch of twenty units
    (300, 40, 2, 5, 1, 40),       # ten units of u, v, sc; wide and low
    (512, 256, 4, 2, 10, 2),
])
@pytest.mark.parametrize("obstacles", [False, True])
def test_bitexact(nx, ny, ngrid, nswpm, nswpp, ncases, obstacles, oracle_built):
    from mgfvm import Solver
    from oracle import OracleCase
    base = _cfg(nx, ny, ngrid, nswpm, nswpp, obstacles)
    cfgs = [base.replace(amuf=1.0 / (20.0 + 3 * k)) for k in range(ncases)]
    with Solver(cfgs) as s:
        s.set_tuning(band_visit=[1] * ngrid)
        kinds = {(k, lv) for k, lv, _ in s.profile_cycle()}
        assert ("smooth_q", 0) in kinds
        s.cycle(2)
        for k in (0, ncases - 1):
            o = OracleCase(cfgs[k])
            o.cycle(3)
            for ig in range(ngrid):
                for f in STATE:
                    assert_bitexact(s.field(k, ig, f), o.get(ig, f), f"case {k} level {ig} {f}")
            o.close()


def test_two_sizes(oracle_built):
    from mgfvm import Solver
    from oracle import OracleCase
    cfgs = [_cfg(200, 120, 2, 2, 10, True), _cfg(96, 144, 2, 2, 10, False)] * 20
    with Solver(cfgs) as s:
        assert ("smooth_q", 0) in {(k, lv) for k, lv, _ in s.profile_cycle()}
        s.cycle(1)
        for k in (0, 1, 39):
            o = OracleCase(cfgs[k])
            o.cycle(2)
            for f in STATE:
                assert_bitexact(s.field(k, 0, f), o.get(0, f), f"case {k} {f}")
            o.close()
