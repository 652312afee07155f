"""mgfvm_rbgs_f64_noalloc takes no device memory, and mgfvm_rbgs_f64 gives the same bits where
the device has no room for its buffer.  (Each in a process of its own: what the library's
pool kept from earlier tests would serve the buffer.)"""
import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

HEAD = """
import ctypes as C, sys
sys.path[:0] = [{tests!r}, {pkg!r}]
import numpy as np, torch
from mgfvm import lib
from mgfvm._lib import check
from test_gpu_raw_tiles import COEFS, _dev, _level, _sweeps
from conftest import assert_bitexact

def run(name, npx, npy, nsw, before=None):
    d, phi = _level(npx, npy, 3)
    t = [_dev(d[k], False) for k in COEFS] + [_dev(phi, False)]
    torch.cuda.synchronize()
    if before:
        before()
    free = torch.cuda.mem_get_info()[0]
    check(getattr(lib(), name)(*(C.c_void_p(x.data_ptr()) for x in t), npx, npy, npx - 1, npy - 1, nsw, None))
    torch.cuda.synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    assert_bitexact(t[6].cpu().numpy().reshape(npy, npx), _sweeps(d, phi, npx - 1, npy - 1, nsw, True), "phi")
    return taken
"""


def _python(body):
    head = HEAD.format(tests=os.path.join(REPO, "tests"), pkg=os.path.join(REPO, "multigrid-fvm_b200"))
    r = subprocess.run([sys.executable, "-c", head + body], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_takes_no_device_memory():
    _python("""
run("mgfvm_rbgs_f64_noalloc", 200, 150, 3)      # loads the kernels of both shapes
run("mgfvm_rbgs_f64_noalloc", 30, 30, 3)
for npx, npy, nsw in ((30, 40, 5), (54, 56, 2), (55, 56, 4), (403, 310, 10), (1026, 1026, 3)):
    assert run("mgfvm_rbgs_f64_noalloc", npx, npy, nsw) == 0, (npx, npy)
""")


def test_no_room_for_the_buffer():
    """All but some 100 MB of the device is taken, the buffer would be 134."""
    _python("""
run("mgfvm_rbgs_f64_noalloc", 200, 150, 3)      # loads the kernels
held = []
def fill():
    torch.cuda.empty_cache()
    for size in (4 << 30, 256 << 20, 64 << 20):
        while torch.cuda.mem_get_info()[0] > size + (48 << 20):
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
n = run("mgfvm_rbgs_f64", 4096, 4096, 5, fill)
assert n == 0, n
held.clear()
torch.cuda.empty_cache()
assert run("mgfvm_rbgs_f64", 4096, 4096, 5) > 0     # with room, the buffer stays in the pool
""")
