"""The tile kernels (assembly, restriction, prolongation: 32 x 8 cells a block) at the edges
of their tiles: grids one cell pair short of, at and beyond whole tiles, a single row of
tiles, odd coarsest levels, obstacles on the tiles' seams, every boundary kind.  The FP64
engine applies the reference's operations in its order whatever the tiling, so the bar is
the oracle's bits (as in test_gpu_parity.py); mixed precision is held to the bits of the
sliced kernels, which form the same FP32 operands from the same FP64 values."""
import numpy as np
import pytest

from cases import TOUCHING
from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

STATE = ["u", "v", "p", "pp", "sc", "su", "resu", "resv", "ressc", "apu", "apv", "cx", "cy", "c"]

# (nx, ny, ngrid): padded 32 x 8 tiles and interior ones, less, whole and more
SIZES = [(4, 4, 2), (30, 6, 2), (32, 8, 3), (34, 10, 2), (62, 14, 2), (64, 16, 4), (66, 18, 2), (96, 40, 3),
         (28, 68, 3)]


def _cfg(nx, ny, ngrid, isolve, kind):
    from mgfvm import configs
    cfg = configs.small(32, ngrid, isolve=isolve, nfx=nx, nfy=ny, xl=nx / ny, yl=1.0)
    if kind == "obstacles" and min(nx, ny) >> (ngrid - 1) >= 4:
        w, h = nx >> (ngrid - 1), ny >> (ngrid - 1)
        obs = [o for o in TOUCHING if o[1] <= w and o[3] <= h] + [(w // 2, w // 2 + 1, h // 2, h // 2)]
        return cfg.replace(ig_obs=ngrid, sc_obs=0.25, obstacles=obs)
    if kind == "mixed_bc":
        return cfg.replace(ibc_xm=3, ibc_ym=3, ibc_xp=2, ibc_yp=2, guess=(0.1, 0.05, 0.2, 0.3))
    return cfg


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("isolve,kind", [(1, "channel"), (2, "obstacles"), (2, "mixed_bc")])
def test_tiles_bitexact(size, isolve, kind, oracle_built):
    from mgfvm import Solver
    from oracle import OracleCase
    cfg = _cfg(*size, isolve, kind)
    with Solver(cfg) as s:
        s.set_tuning(pp_level=[1] * cfg.ngrid)      # no one-launch visits: every level assembled by tiles
        o = OracleCase(cfg)
        s.cycle(2)
        o.cycle(2)
        for op in ("restrict", "prolong"):          # and as single routines
            s.op(op, 0)
            o.op(op, 0)
        for ig in range(cfg.ngrid):
            for f in STATE:
                if f in ("su", "pp") and ig == 0:
                    continue                        # the restriction's own coefficient sets in the oracle
                assert_bitexact(s.field(0, ig, f), o.get(ig, f), f"{size} {kind} level {ig} {f}")
        o.close()


@pytest.mark.parametrize("size", [(64, 48, 3), (98, 54, 2)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("isolve", [1, 2])
def test_tiles_mixed_precision_equal_sliced(size, isolve):
    from mgfvm import Solver
    cfgs = [_cfg(*size, isolve, "obstacles"), _cfg(*size, isolve, "channel")]
    runs = []
    for slices in (0, 3):
        with Solver(cfgs, precision="mixed") as s:
            s.set_tuning(asm_slices=[slices] * 3, restrict_slices=[slices] * 3)
            s.cycle(4)
            runs.append([[s.field(k, ig, f) for ig in range(c.ngrid) for f in ("u", "v", "p", "sc", "resu", "cx")]
                         for k, c in enumerate(cfgs)])
    for a, b in zip(runs[0], runs[1]):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
