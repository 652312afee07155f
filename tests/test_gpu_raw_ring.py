"""The raw smoothers write the cells they sweep and no others: what another stream stores in
the cells round the extents while a call runs is still there after it."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_bitexact
from test_gpu_raw_tiles import COEFS, _call, _dev, _level, _sweeps

pytestmark = pytest.mark.gpu


# a call of some milliseconds, in one launch in place and in many through a buffer
@pytest.mark.parametrize("gs", [True, False])
@pytest.mark.parametrize("npx,npy,nx,ny,nsw", [
    (64, 60, 31, 40, 12000),
    (420, 300, 400, 280, 400),
])
def test_ring_is_left_alone(gs, npx, npy, nx, ny, nsw):
    import torch
    d, phi = _level(npx, npy, 11)
    # the sweeps read the ring and take nothing from it
    d["aw"][:, 1] = 0.0
    d["ae"][:, nx - 1] = 0.0
    d["as"][1, :] = 0.0
    d["an"][ny - 1, :] = 0.0
    inside = np.zeros((npy, npx), dtype=bool)
    inside[1:ny, 1:nx] = True
    co = [_dev(d[k], False) for k in COEFS]
    t, scratch = _dev(phi, False), _dev(phi, False)
    outside = torch.from_numpy(~inside).cuda().reshape(-1)
    sides = [t.view(npy, npx)[s] for s in (np.s_[0, :], np.s_[ny:, :], np.s_[1:ny, 0], np.s_[1:ny, nx:])]
    a, b = torch.cuda.Stream(), torch.cuda.Stream(priority=-1)
    with torch.cuda.stream(b):
        for s in sides:
            s.fill_(3.0)        # (loads the kernels the second round needs)
    torch.cuda.synchronize()
    _call(gs, co, t, scratch, npx, npy, nx, ny, nsw, C.c_void_p(a.cuda_stream))
    with torch.cuda.stream(b):
        for s in sides:
            s.fill_(7.0)
    torch.cuda.synchronize()
    assert bool((t[outside] == 7.0).all())
    want = _sweeps(d, phi, nx, ny, nsw, gs)
    assert_bitexact(t.cpu().numpy().reshape(npy, npx)[1:ny, 1:nx], want[1:ny, 1:nx], "phi")
