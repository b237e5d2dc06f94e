"""A program may end its CUDA context (cudaDeviceReset) and begin another: a
context of the library made then, and the allocation-free solve, work as the
first ones did.  In child processes, which the reset leaves without effect on
other tests."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_RESET = r"""
import ctypes, sys
sys.path.insert(0, %r)
import numpy as np
import lu2_b200 as L

class Dev:
    def __init__(self, ptr): self.ptr = ptr
    def data_ptr(self): return self.ptr

rt = ctypes.CDLL("libcudart.so.12")
rng = np.random.default_rng(1)

def solve(n, noalloc):
    ld = L.device_ld(n)
    host = np.zeros((n, ld))
    host[:, :n + 1] = rng.uniform(-0.5, 0.5, (n, n + 1))
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(host.nbytes)) == 0
    assert rt.cudaMemcpy(p, host.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(host.nbytes), 1) == 0
    if noalloc:
        assert L.load().lu2gpu_lusolve_noalloc(n, 1, p.value, ld, 64, 1, None, None) == 0, L._lib.last_error()
    else:
        c = L.Context(0)
        assert c.lusolve(p.value, n, ld, 64) == 0
        c.close()
    out = np.zeros_like(host)
    assert rt.cudaMemcpy(out.ctypes.data_as(ctypes.c_void_p), p, ctypes.c_size_t(host.nbytes), 2) == 0
    assert rt.cudaFree(p) == 0
    x, a, b = out[:, n], host[:, :n], host[:, n]
    h = np.abs(a @ x - b).max() / (2.0 ** -53 * (np.abs(a).sum(1).max() * np.abs(x).max() + np.abs(b).max()) * n)
    assert h < 16, h

order = sys.argv[1].split(",")
solve(500, order[0] == "noalloc")
for step in order:
    assert rt.cudaDeviceReset() == 0
    solve(700, step == "noalloc")
print("solved after a reset")
"""


@pytest.mark.parametrize("steps", ["context", "context,context", "noalloc", "noalloc,context,noalloc"])
def test_solves_after_a_device_reset(steps):
    r = subprocess.run([sys.executable, "-c", _RESET % ROOT, steps], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and "solved after a reset" in r.stdout, r.stdout + r.stderr
