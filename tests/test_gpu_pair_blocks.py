"""The pair smoother's two block sizes against the oracle, bit for bit: batches whose half-size
CTAs just have an SM each and one case more, both smoothers, unequal launches."""
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "p", "pp", "sc", "su", "apu", "apv"]


@pytest.mark.parametrize("isolve", [1, 2])
@pytest.mark.parametrize("nx,ny,ncases,nswpm,nswpp", [
    (64, 64, 4, 2, 10),      # p' by Jacobi: 36 tiles a case, 144 CTAs
    (64, 64, 5, 2, 10),      # 180
    (152, 56, 3, 3, 7),
    (70, 66, 1, 1, 13),      # launches of unequal length
    (45, 47, 2, 2, 4),       # odd rows
])
def test_bitexact(isolve, nx, ny, ncases, nswpm, nswpp, oracle_built):
    from mgfvm import Solver, configs
    from oracle import OracleCase
    cfgs = [configs.small(32, 1, isolve=isolve, nfx=nx, nfy=ny, xl=nx / ny, yl=1.0, nswpm=nswpm, nswpp=nswpp,
                          amuf=1.0 / (20.0 + 3 * k), ig_obs=1, sc_obs=0.2, obstacles=[(9, 20, 11, 25)]) for k in range(ncases)]
    with Solver(cfgs) as s:
        s.cycle(4)
        for k in (0, ncases - 1):
            o = OracleCase(cfgs[k])
            o.cycle(4)
            for f in STATE:
                assert_bitexact(s.field(k, 0, f), o.get(0, f), f"case {k} {f}")
            o.close()
