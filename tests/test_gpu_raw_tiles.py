"""The raw smoothers by tiles (mgfvm_rbgs_f64, mgfvm_jacobi_f64) against sweeps restated in
numpy, bit for bit: levels that fit one tile and a cell more, several launches of equal and
unequal sweeps, extents smaller than the level, arrays at an odd 8-byte offset (no paired
loads), and calls on a stream that is being captured (which get no buffer of their own)."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

COEFS = ("aw", "ae", "as", "an", "ap", "su")


def _level(npx, npy, seed):
    rng = np.random.default_rng(seed)
    d = {k: rng.uniform(0.05, 1.0, (npy, npx)) for k in ("aw", "ae", "as", "an")}
    d["ap"] = d["aw"] + d["ae"] + d["as"] + d["an"] + rng.uniform(0.0, 0.5, (npy, npx))
    d["su"] = rng.standard_normal((npy, npx)) * 10.0 ** rng.integers(-200, 3, (npy, npx))
    d["ap"][npy // 3, npx // 2] = 1.0e30        # a solid cell
    phi = rng.standard_normal((npy, npx))
    phi[rng.random((npy, npx)) < 0.3] = 0.0
    return d, phi


def _sweeps(d, phi, nx, ny, nsw, gs):
    p = phi.copy()
    c, w, e = np.s_[1:ny, 1:nx], np.s_[1:ny, 0:nx - 1], np.s_[1:ny, 2:nx + 1]
    s, n = np.s_[0:ny - 1, 1:nx], np.s_[2:ny + 1, 1:nx]
    jj, ii = np.mgrid[1:ny, 1:nx]
    for _ in range(nsw):
        for colour in ((0, 1) if gs else (None,)):
            x = d["aw"][c] * p[w] + d["ae"][c] * p[e] + d["as"][c] * p[s] + d["an"][c] * p[n] + d["su"][c]
            if gs:
                p[c] = np.where((ii + jj) % 2 == colour, x / d["ap"][c], p[c])
            else:
                p[c] = x / (d["ap"][c] + 1.0e-30)
    return p


def _dev(a, odd):
    import torch
    t = torch.zeros(a.size + 2, dtype=torch.float64, device="cuda")
    v = t[1 if odd else 0:][:a.size]
    v.copy_(torch.from_numpy(a.reshape(-1)))
    return v


def _call(gs, co, phi, scratch, npx, npy, nx, ny, nsw, stream=None):
    from mgfvm import lib
    from mgfvm._lib import check
    p = [C.c_void_p(t.data_ptr()) for t in (*co, phi)]
    if gs:
        check(lib().mgfvm_rbgs_f64(*p, npx, npy, nx, ny, nsw, stream))
    else:
        check(lib().mgfvm_jacobi_f64(*p, C.c_void_p(scratch.data_ptr()), npx, npy, nx, ny, nsw, stream))


@pytest.mark.parametrize("gs", [True, False])
@pytest.mark.parametrize("npx,npy,nx,ny,nsw,odd", [
    (54, 56, 53, 55, 7, False),       # one region of the GS tiles, whole
    (55, 56, 54, 55, 7, False),       # a column more, odd rows
    (54, 57, 53, 56, 8, True),
    (32, 64, 31, 63, 6, False),       # one tile of the Jacobi pairs, whole
    (33, 64, 32, 63, 6, True),
    (3, 3, 2, 2, 12, False),          # one cell
    (300, 4, 299, 2, 12, False),      # one row
    (4, 300, 2, 299, 11, True),       # one column
    (128, 96, 101, 64, 12, False),    # extents inside the level
    (127, 96, 101, 64, 11, False),
    (403, 310, 402, 309, 10, False),
    (610, 512, 609, 511, 40, False),  # many launches
])
def test_bitexact(gs, npx, npy, nx, ny, nsw, odd):
    import torch
    d, phi = _level(npx, npy, npx * 1000 + nsw)
    want = _sweeps(d, phi, nx, ny, nsw, gs)
    co = [_dev(d[k], odd) for k in COEFS]
    t, scratch = _dev(phi, odd), _dev(phi * 0.0 + 3.0, odd)
    _call(gs, co, t, scratch, npx, npy, nx, ny, nsw)
    torch.cuda.synchronize()
    assert_bitexact(t.cpu().numpy().reshape(npy, npx), want, "phi")
    for k, c in zip(COEFS, co):
        assert_bitexact(c.cpu().numpy().reshape(npy, npx), d[k], k)


@pytest.mark.parametrize("gs", [True, False])
def test_capture(gs):
    import torch
    npx, npy, nsw = 203, 150, 9
    d, phi = _level(npx, npy, 5)
    co = [_dev(d[k], False) for k in COEFS]
    t, scratch = _dev(phi, False), _dev(phi, False)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _call(gs, co, t, scratch, npx, npy, npx - 1, npy - 1, nsw, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert_bitexact(t.cpu().numpy().reshape(npy, npx), _sweeps(d, phi, npx - 1, npy - 1, 2 * nsw, gs), "phi")


@pytest.mark.parametrize("npx,npy", [(3, 3), (400, 380), (401, 381), (390, 392), (1201, 700)])
def test_masserror(npx, npy):
    import torch
    from mgfvm import lib
    from mgfvm._lib import check
    rng = np.random.default_rng(npx)
    ax, ay, u, v = (rng.standard_normal((npy, npx)) for _ in range(4))
    c = np.s_[1:-1, 1:-1]
    div = ax[c] * u[c] - ax[c] * u[1:-1, :-2] + ay[c] * v[c] - ay[c] * v[:-2, 1:-1]
    t = [_dev(a, False) for a in (u, v, ax, ay, u * 0 + 5.0, u * 0 + 7.0)]
    err = torch.zeros(1, dtype=torch.float64, device="cuda")
    partials = torch.zeros(lib().mgfvm_masserror_scratch_doubles(npx, npy), dtype=torch.float64, device="cuda")
    for _ in range(2):
        check(lib().mgfvm_masserror_f64(*(C.c_void_p(x.data_ptr()) for x in t), npx, npy, C.c_void_p(err.data_ptr()),
                                        C.c_void_p(partials.data_ptr()), None))
        torch.cuda.synchronize()
        su, pp = (x.cpu().numpy().reshape(npy, npx) for x in t[4:])
        assert_bitexact(su[c], -div, "su")
        assert np.all(pp[c] == 0.0) and su[0, 0] == 5.0 and pp[-1, -1] == 7.0
        # sums of n terms differ by at most n roundings, far fewer in a tree
        np.testing.assert_allclose(err.item(), np.abs(div).sum(), rtol=1e-13)
