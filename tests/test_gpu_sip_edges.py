"""cfd_sip_solve (one cooperative launch per 256 iterations) at the edges of its forms: the
smallest grids, a grid one column over a tile, more tiles than SMs, a solve longer than one
launch, calls from two threads on streams of their own. Against the sparse direct solution, at
the bar of tests/test_gpu_seam.py."""
import ctypes
import threading

import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu


def _system(kind, n0, n1, seed=3):
    from oracle import oracle
    from tests.test_gpu_seam import SIP_ORDER
    g = ogrid(n0, n1, ar=1.5, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.12)
    coefs = [oracle.OracleCase(g, Re=100.0, dt=2e-3).field(k) for k in SIP_ORDER]
    rng = np.random.default_rng(seed)
    phi0 = rng.standard_normal((n1, n0))
    if kind == "ogrid":
        phi0[:, -1] = phi0[:, 0]
    return g, coefs, phi0, rng.standard_normal((n1, n0)), int(kind == "ogrid")


def _residual(coefs, phi, q, per):
    """|q - A phi| and |A| |phi| summed over the unknown cells."""
    offs = ((0, 0), (1, 0), (0, -1), (0, 1), (-1, 0), (1, -1), (-1, -1), (1, 1), (-1, 1))
    n1, n0 = q.shape
    P = n0 - 1 if per else n0
    r, size = q[:, :P].copy(), np.abs(q[:, :P])
    for a, (di, dj) in zip(coefs, offs):
        t = a[:, :P] * np.roll(phi[:, :P], (-dj, -di), (0, 1))
        r -= t
        size += np.abs(t)
    sl = (slice(1, -1), slice(None) if per else slice(1, -1))
    return np.abs(r[sl]).sum(), size[sl].sum()


@pytest.mark.parametrize("kind,n0,n1", [("ogrid", 8, 6), ("cavity", 8, 7), ("ogrid", 34, 19), ("cavity", 35, 18),
                                        ("ogrid", 289, 305), ("cavity", 321, 273)])
def test_edges(kind, n0, n1):
    """The rule the solve promises: the L1 residual below tol times the first. The recurrence's
    residual and the true one part by rounding of the matrix products, a few units in the last
    place of |A| |phi| per product, at most 2 x 2 products an iteration. On the small grids,
    whose condition numbers stay below 1e3, the solution too."""
    from tests.test_gpu_seam import direct_solve, sip_gpu
    g, coefs, phi0, q, per = _system(kind, n0, n1)
    rc, phi, iters = sip_gpu(g, coefs, phi0, q, per, tol=1e-13)
    assert rc == 0
    first, size0 = _residual(coefs, phi0, q, per)
    last, size = _residual(coefs, phi, q, per)
    assert last <= 1e-13 * first + 16 * 2.3e-16 * (iters + 1) * (size + size0)
    if n0 * n1 < 1000:
        ref = direct_solve(coefs, phi0, q, per)
        assert np.linalg.norm(phi - ref) / np.linalg.norm(ref) < 1e-10
    np.testing.assert_array_equal(phi[[0, -1]], phi0[[0, -1]])


def test_more_iterations_than_one_launch_takes():
    """A grid without a coarser level at a tolerance no residual meets: 256 + 44 iterations."""
    from tests.test_gpu_seam import direct_solve, sip_gpu
    g, coefs, phi0, q, per = _system("ogrid", 46, 94)
    rc, phi, iters = sip_gpu(g, coefs, phi0, q, per, tol=0.0, maxit=300)
    assert rc == -5 and iters == 300  # CFD_E_MAXITER
    ref = direct_solve(coefs, phi0, q, per)
    assert np.linalg.norm(phi - ref) / np.linalg.norm(ref) < 1e-10


def test_two_threads_on_their_own_streams():
    import torch
    from cfd_solver_b200 import _lib
    g, coefs, phi0, q, per = _system("ogrid", 65, 49)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in coefs]
    ptrs = (ctypes.c_void_p * 9)(*[t.data_ptr() for t in dev])
    qd, p0 = torch.from_numpy(q).cuda(), torch.from_numpy(phi0).cuda()
    torch.cuda.synchronize()

    def solve(stream):
        with torch.cuda.stream(stream):
            phi, it = p0.clone(), ctypes.c_int(0)
            rc = _lib.lib().cfd_sip_solve(g.n0, g.n1, per, ptrs, ctypes.c_void_p(phi.data_ptr()),
                                          ctypes.c_void_p(qd.data_ptr()), 1e-8, 100, ctypes.byref(it),
                                          ctypes.c_void_p(stream.cuda_stream))
            return rc, it.value, phi.cpu().numpy()

    alone = solve(torch.cuda.current_stream())
    got = [[] for _ in range(2)]

    def work(k):
        s = torch.cuda.Stream()
        for _ in range(10):
            got[k].append(solve(s))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in got[0] + got[1]:
        assert r[:2] == alone[:2]
        np.testing.assert_array_equal(r[2], alone[2])
