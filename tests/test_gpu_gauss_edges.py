"""cfd_gauss_solve (one cooperative launch per solve) at the edges of its forms: the smallest
grids, one cell more or less than a multiple of a CTA's 256, more cells than the resident
threads (each thread then has several), a solve longer than one launch's 512 sweeps, a
residual that is not finite, and calls from two threads on streams of their own. Against the
oracle's tightly converged gauss(), at the bar of tests/test_gpu_seam.py."""
import ctypes
import threading

import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu


def _grid(kind, n0, n1):
    return ogrid(n0, n1, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.1)


@pytest.mark.parametrize("kind,n0,n1", [
    ("ogrid", 8, 6), ("cavity", 8, 7),
    ("ogrid", 33, 10),   # 32 x 8 = 256 cells
    ("ogrid", 258, 3 + 3), ("cavity", 19, 17),  # 257 x 4 = 1028, 17 x 15 = 255
    ("ogrid", 401, 402),  # 160,000 cells: more than the resident threads
])
def test_edges(kind, n0, n1):
    from cfd_solver_b200 import _lib
    from tests.test_gpu_seam import gpu_solve, system
    g = _grid(kind, n0, n1)
    coefs, phi0, q, ref = system(g, "u", fix_T=1)
    phi, _ = gpu_solve(_lib.lib().cfd_gauss_solve, g, coefs, phi0, q, int(kind == "ogrid"), tol=1e-11)
    sl = (slice(1, -1), slice(None)) if kind == "ogrid" else (slice(1, -1), slice(1, -1))
    assert np.linalg.norm(phi[sl] - ref[sl]) / np.linalg.norm(ref[sl]) < 1e-10
    np.testing.assert_array_equal(phi[[0, -1]], phi0[[0, -1]])
    if kind == "ogrid":
        np.testing.assert_array_equal(phi[1:-1, -1], phi[1:-1, 0])
    else:
        np.testing.assert_array_equal(phi[:, [0, -1]], phi0[:, [0, -1]])


def _call(coefs, phi0, q, periodic, tol, maxit, stream=None):
    import torch
    from cfd_solver_b200 import _lib
    n1, n0 = phi0.shape
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in coefs]
    ptrs = (ctypes.c_void_p * 25)(*[t.data_ptr() for t in dev])
    phi, qd = torch.from_numpy(phi0.copy()).cuda(), torch.from_numpy(np.ascontiguousarray(q)).cuda()
    torch.cuda.synchronize()
    sweeps = ctypes.c_int(0)
    rc = _lib.lib().cfd_gauss_solve(n0, n1, periodic, ptrs, ctypes.c_void_p(phi.data_ptr()),
                                    ctypes.c_void_p(qd.data_ptr()), tol, maxit, ctypes.byref(sweeps),
                                    ctypes.c_void_p(stream.cuda_stream) if stream else None)
    torch.cuda.synchronize()
    return rc, sweeps.value, phi.cpu().numpy()


def test_more_sweeps_than_one_launch_takes():
    from tests.test_gpu_seam import system
    coefs, phi0, q, ref = system(_grid("ogrid", 33, 25), "u", fix_T=1)
    rc, sweeps, phi = _call(coefs, phi0, q, 1, 1e-300, 1301)
    assert rc == -5 and sweeps == 1300  # CFD_E_MAXITER after 512 + 512 + 276 sweeps
    assert np.linalg.norm(phi[1:-1] - ref[1:-1]) / np.linalg.norm(ref[1:-1]) < 1e-10


def test_residual_not_finite_is_reported():
    from tests.test_gpu_seam import system
    coefs, phi0, q, _ = system(_grid("cavity", 33, 29), "u", fix_T=1)
    q = q.copy()
    q[5, 7] = np.nan
    assert _call(coefs, phi0, q, 0, 1e-8, 100)[0] == -4  # CFD_E_DIVERGED


def test_two_threads_on_their_own_streams():
    import torch
    from tests.test_gpu_seam import system
    coefs, phi0, q, _ = system(_grid("ogrid", 65, 49), "u", fix_T=1)
    alone = _call(coefs, phi0, q, 1, 1e-8, 400)
    got = [[] for _ in range(2)]

    def work(k):
        s = torch.cuda.Stream()
        for _ in range(10):
            got[k].append(_call(coefs, phi0, q, 1, 1e-8, 400, s))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in got[0] + got[1]:
        assert r[:2] == alone[:2]
        np.testing.assert_array_equal(r[2], alone[2])
