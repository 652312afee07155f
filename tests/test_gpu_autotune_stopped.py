"""The autotuner times running cycles, also of cases that an earlier solve has stopped, and
leaves the state and the history of those as they were."""
import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


def test_autotune_after_a_stop():
    from mgfvm import Solver, configs
    cfgs = [configs.small(256, 5, isolve=2, amuf=1.0 / (20.0 + k)) for k in range(2)]
    with Solver(cfgs) as s:
        s.cycle(20)
        s.cycle(20)
        running = s.last_elapsed_ms / 20
        s.reset()
        assert list(s.solve(9, 1e30)) == [2, 2]       # the fixed-point rule stops both
        before = [[s.field(k, 0, f) for f in ("u", "v", "p", "sc")] + [s.history(k)[0]] for k in range(2)]
        t_before, t_after, _ = s.autotune(5)
        # a cycle of stopped cases takes a quarter of a running one
        assert t_before > 0.7 * running and t_after <= t_before, (t_before, t_after, running)
        for k in range(2):
            for a, b in zip(before[k], [s.field(k, 0, f) for f in ("u", "v", "p", "sc")] + [s.history(k)[0]]):
                assert_bitexact(b, a, f"case {k}")
        s.cycle(1)
        assert len(s.history(0)[0]) == 3
