"""The seams after the host program has reset the device.

cudaDeviceReset() ends the process's own context and with it whatever the library kept in it (the
scratch pool, the address of the static scratch); the next call starts again from nothing. Each
case runs in a process of its own.
"""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
PROGRAM = r"""
import ctypes, glob, os, sys
import numpy as np
import torch
from cfd_solver_b200 import _lib
L = _lib.lib()
rt = ctypes.CDLL(glob.glob(os.path.join(os.path.dirname(torch.__file__), "../nvidia/cuda_runtime/lib/libcudart.so*"))[0])
n = 129
def up(a):
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes), 1) == 0
    return p
def call(seam):
    rng = np.random.default_rng(5)
    off = up(-0.03 * rng.random((n, n))); ap = up(2.0 + rng.random((n, n)))
    phi = up(np.zeros((n, n))); q = up(rng.standard_normal((n, n)))
    k = 9 if seam == "sip" else 25
    co = (ctypes.c_void_p * k)(ap.value, *[off.value] * (k - 1))
    it = ctypes.c_int()
    f = {"gauss": L.cfd_gauss_solve, "noalloc": L.cfd_gauss_solve_noalloc, "sip": L.cfd_sip_solve}[seam]
    rc = f(n, n, 0, co, phi, q, ctypes.c_double(1e-9), 200, ctypes.byref(it), None)
    assert rc == 0 and it.value > 1, (rc, it.value)
    out = np.empty((n, n))
    assert rt.cudaMemcpy(out.ctypes.data_as(ctypes.c_void_p), phi, ctypes.c_size_t(out.nbytes), 2) == 0
    return out
first = call(sys.argv[1])
for _ in range(3):
    assert rt.cudaDeviceReset() == 0
    np.testing.assert_array_equal(call(sys.argv[1]), first)
print("same")
"""


@pytest.mark.parametrize("seam", ["gauss", "sip", "noalloc"])
def test_seam_after_a_device_reset(seam):
    r = subprocess.run([sys.executable, "-c", PROGRAM, seam], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
