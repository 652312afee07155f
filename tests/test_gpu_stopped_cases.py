"""Cases that have stopped cost their launches and little else, and are left out of the table
of tiles wherever they lie in it."""
import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


def _cfgs(n, ncases, isolve=2, **kw):
    from mgfvm import configs
    return [configs.small(n, 5, isolve=isolve, nfy=n, amuf=1.0 / (20.0 + k), **kw) for k in range(ncases)]


# A running cycle is the stopped one's launches (1.2 to 1.6 us each, and the blocks' own start
# in large batches) plus the work.  Measured: 0.12, 0.26, 0.20 and 0.28 of a running one; half
# as much again is allowed.  With every block reading its data before the flag: 0.66, 0.50,
# 0.59 and 0.52.
@pytest.mark.parametrize("n,ncases,isolve,precision,most", [
    (256, 64, 2, "fp64", 0.20),
    (256, 2, 2, "fp64", 0.40),
    (256, 12, 2, "mixed", 0.32),
    (192, 3, 1, "fp64", 0.42),
])
def test_time(n, ncases, isolve, precision, most):
    from mgfvm import Solver
    cycles = 64
    with Solver(_cfgs(n, ncases, isolve), precision=precision, sync_every=cycles) as s:
        run, mixed = [], []
        for _ in range(4):
            s.reset()
            s.cycle(cycles)
            run.append(s.last_elapsed_ms)
            s.reset()
            # the fixed-point rule stops every case after its second cycle; the rest of the
            # chunk is queued by then
            assert list(s.solve(cycles, 1e30)) == [2] * ncases
            mixed.append(s.last_elapsed_ms)
        running = min(run) / cycles
        stopped = (min(mixed) - 2 * running) / (cycles - 2)
        assert stopped < most * running, (stopped, running)


def test_tiles_past_the_flags_kept():
    """More tiles a CTA than it keeps flags for (384): stopped and running cases among the rest."""
    from mgfvm import Solver, configs
    cfgs = [configs.small(1024, 1, isolve=2, nswpp=4, amuf=1.0 / (20.0 + k), convergence=(1e30, 1e-30)[k % 2])
            for k in range(44)]
    with Solver(cfgs) as s:
        assert list(s.solve(2)) == [1, 2] * 22
        for k in (0, 1, 40, 41, 42, 43):
            with Solver(cfgs[k].replace(convergence=1e-6)) as one:
                one.cycle(1 + k % 2)
                for f in ("u", "v", "p", "sc"):
                    assert_bitexact(s.field(k, 0, f).view(np.int64), one.field(0, 0, f).view(np.int64), f"case {k} {f}")
