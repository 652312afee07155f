"""The adjoint's grouped passes where their shape changes: a program too long for shared
memory, a level of more cells than the small CTA is for, one column of cells more than the
workers, Jacobi with an odd sweep count.  The bar is the forward mode's gradient (the same
derivatives, accumulated in another order): 1e-10 of its largest entry, the bar the other
adjoint tests hold the two to."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ngrid,isolve,nswpm,nswpp", [
    (16, 16, 2, 2, 2, 200),    # 836 phases
    (144, 144, 2, 2, 1, 4),    # 21316 cells: the large CTA
    (66, 130, 1, 2, 2, 3),     # 4290 cells of a colour over 4096 workers
    (34, 18, 2, 1, 3, 5),
])
def test_equals_forward_mode(nx, ny, ngrid, isolve, nswpm, nswpp):
    from mgfvm import Solver, configs, gradient
    w, h = nx >> (ngrid - 1), ny >> (ngrid - 1)
    cfg = configs.small(32, ngrid, isolve=isolve, nfx=nx, nfy=ny, xl=nx / ny, yl=1.0, nswpm=nswpm, nswpp=nswpp,
                        ig_obs=ngrid, sc_obs=0.3, guess=(0.1, 0.0, 0.0, 0.2),
                        obstacles=[(w // 2, w // 2 + 1, h // 2, h // 2 + 1), (w // 4, w // 4, h // 4, h // 4)])
    prof = 1.0 + 0.1 * np.random.default_rng(3).standard_normal(ny)
    j, g_in, g_a, g_p = gradient(cfg, prof, cycles=2)
    with Solver(cfg) as s:
        s.set_inlet_profile(0, prof)
        s.adjoint(2)
        ja, a_in, a_a, a_p = s.adjoint_gradient(0)
    top = max(np.abs(g_in).max(), abs(g_a), abs(g_p))
    assert abs(ja - j) <= 1e-12 * abs(j)
    assert np.abs(a_in - g_in).max() <= 1e-10 * top
    assert abs(a_a - g_a) <= 1e-10 * top and abs(a_p - g_p) <= 1e-10 * top
