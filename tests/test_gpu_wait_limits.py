"""Counter barriers that run out: the grid-form team kernel, the sip9p() and gauss() seams.

Their waits poll a limited number of times, which the launch carries as an argument. With a limit
of zero every CTA gives up at its first barrier, without waiting for anything: the call fails
with CFD_E_CUDA, a team launch queued behind leaves the batch as it is, and the next call with
the usual limit gives the usual result. (A cluster's hardware barrier has no limit: its CTAs are
resident together and all of them arrive.)
"""
import ctypes

import numpy as np
import pytest

from cfd_solver_b200.grid import cavity

pytestmark = pytest.mark.gpu

E_CUDA = -2
POLLS = ctypes.c_uint(1 << 24)
NONE = ctypes.c_uint(0)


def _batch(n, mixed):
    from cfd_solver_b200.solver import Batch, case_params
    g = cavity(193, 193, skew=0.1)  # 72 tiles: a share of the grid
    return Batch([g] * n, [case_params(g, Re=200.0, dt=1e-3, precision=mixed)] * n)


def _image(b):
    img = np.zeros(b.state_bytes() // 8)
    b.get_state(img)
    return img.view(np.int64)


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("n", [1, 2])
def test_team_barrier_that_runs_out(n, mixed):
    from cfd_solver_b200 import _lib
    L = _lib.lib()
    with _batch(n, mixed) as b:
        b.step(2)
        ref = _image(b)
    with _batch(n, mixed) as b:
        assert L.cfd_internal_team_steps(b.h, 2, POLLS) == 0
        np.testing.assert_array_equal(_image(b), ref)
        assert L.cfd_internal_team_steps(b.h, 4, NONE) == E_CUDA
        assert b"bounded wait" in L.cfd_last_error()
        work = b.work()
        # queued behind the failure: no step is taken, and the failure is still reported
        assert L.cfd_internal_team_steps(b.h, 2, POLLS) == E_CUDA
        assert b.work() == work
        with pytest.raises(_lib.CfdError, match="bounded wait"):
            b.step(40)
        assert b.work() == work
    with _batch(n, mixed) as b:  # the device is as good as before
        b.step(2)
        np.testing.assert_array_equal(_image(b), ref)


@pytest.mark.parametrize("seam", ["gauss", "sip"])
@pytest.mark.parametrize("n", [8, 65, 257])  # one tile, a few, the chip
def test_seam_barrier_that_runs_out(seam, n):
    import torch
    from cfd_solver_b200 import _lib
    L = _lib.lib()
    f = {"gauss": L.cfd_internal_gauss_solve, "sip": L.cfd_internal_sip_solve}[seam]
    k = 25 if seam == "gauss" else 9
    rng = np.random.default_rng(n)
    off = torch.from_numpy(-0.03 * rng.random((n, n))).cuda()
    ap = torch.from_numpy(2.0 + rng.random((n, n))).cuda()
    q = torch.from_numpy(rng.standard_normal((n, n))).cuda()
    coef = (ctypes.c_void_p * k)(ap.data_ptr(), *[off.data_ptr()] * (k - 1))

    def call(polls):
        phi, it = torch.zeros_like(q), ctypes.c_int()
        torch.cuda.synchronize()
        rc = f(n, n, 0, coef, ctypes.c_void_p(phi.data_ptr()), ctypes.c_void_p(q.data_ptr()), ctypes.c_double(1e-9), 200,
               ctypes.byref(it), None, polls)
        torch.cuda.synchronize()
        return rc, phi.cpu().numpy()
    rc, ref = call(POLLS)
    assert rc == 0 and np.any(ref)
    rc, _ = call(NONE)
    assert rc == E_CUDA and b"wait" in L.cfd_last_error() and b"timed out" in L.cfd_last_error()
    rc, again = call(POLLS)
    assert rc == 0
    np.testing.assert_array_equal(again, ref)
