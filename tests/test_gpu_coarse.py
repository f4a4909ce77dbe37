"""The coarsest multigrid level's solve at the edges of its forms.

A grid whose sides do not halve has one level, so the whole preconditioner is the coarsest
level's sweeps. They run with one, two or four unknowns per thread in registers (1024
threads), or re-read them in every pass above that; every size here is one side or the other of
an edge. The solve must reach the sparse direct solution (tests/test_gpu_seam.py's bar).
"""
import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n0,n1", [
    ("ogrid", 46, 24),    # 45 x 22 = 990 unknowns: one per thread (odd width: six colours)
    ("ogrid", 46, 26),    # 45 x 24 = 1080: two
    ("ogrid", 46, 48),    # 45 x 46 = 2070: four
    ("ogrid", 46, 94),    # 45 x 92 = 4140: stencils re-read in every pass
    ("ogrid", 132, 130),  # 131 x 128, x of 130 x 137 words: x in its plane as well
    ("cavity", 34, 34),   # 32 x 32 = 1024: one (four colours)
    ("cavity", 66, 66),   # 64 x 64 = 4096: four, x of 66 x 70 words
    ("cavity", 10, 512),  # 8 x 510 = 4080 unknowns, x of 512 x 14 words: two, four or re-read
])
def test_single_level_solve_matches_direct_solve(kind, n0, n1):
    from oracle import oracle
    from tests.test_gpu_seam import SIP_ORDER, direct_solve, sip_gpu
    g = ogrid(n0, n1, ar=1.5, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.1)
    periodic = int(kind == "ogrid")
    coefs = [oracle.OracleCase(g, Re=100.0, dt=2e-3).field(k) for k in SIP_ORDER]
    rng = np.random.default_rng(n0 * n1)
    phi0 = np.zeros((n1, n0))
    q = rng.standard_normal((n1, n0))
    rc, phi, iters = sip_gpu(g, coefs, phi0, q, periodic, tol=1e-12, maxit=2000)
    assert rc == 0, (rc, iters)
    ref = direct_solve(coefs, phi0, q, periodic)
    err = np.linalg.norm(phi - ref) / np.linalg.norm(ref)
    assert err < 1e-10, (err, iters)
