"""Every form of the coarsest level's solve at the edges of its range, in both kernels that run it.

A grid whose sides do not halve has one level, so the preconditioner is that level's Gauss-Seidel
sweeps alone. k_mg_coarse (1024 threads; the step launch by launch) and the team kernel (512
threads; the sip9p() seam) choose a form by the unknowns n, the points of the largest colour m
and the words w that x takes with its margins:

               k_mg_coarse      team kernel
  small        n <= 1024        n <= 512        a point per thread
  regs 1       m <= 1024        m <= 512        a point of each colour per thread
  regs 2       -                m <= 1024       two
  stream       w <= 12000       w <= 12000      stencils re-read, x in shared memory
  stream, far  above            above           x in its plane

One BiCGStab iteration applies the preconditioner twice and nothing else: its result is compared
with the same iteration in 64 bits with the sweeps written out by colour.

Bar: a sweep's update has some 20 FP32 roundings of 6e-8 each, and the errors of the 12 sweeps
add up (Gauss-Seidel does not amplify them): below 12 * 20 * 6e-8 = 1.5e-5 of x, 1e-4 with the
two applications and the step lengths. A point missed, doubled or taken in another colour's turn
is off by a tenth or more at that point.
"""
import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid
from tests.test_gpu_seam import SIP_ORDER, sip_gpu

pytestmark = pytest.mark.gpu

BAR = 1e-4
SWEEPS = 12
OFFSETS = {"ae": (1, 0), "aw": (-1, 0), "an": (0, 1), "as": (0, -1), "ane": (1, 1), "anw": (-1, 1), "ase": (1, -1),
           "asw": (-1, -1)}

# (kind, n0, n1): n, m, w; the form in the team kernel / in k_mg_coarse
GRIDS = [
    ("cavity", 18, 34),   # n 512: small / small
    ("ogrid", 28, 21),    # n 513, m 130 (odd width): regs 1 / small
    ("cavity", 34, 34),   # n 1024: regs 1 / small
    ("ogrid", 42, 27),    # n 1025, m 260 (odd width): regs 1 / regs 1
    ("cavity", 66, 34),   # m 512: regs 1 / regs 1
    ("cavity", 56, 40),   # m 513: regs 2 / regs 1
    ("cavity", 66, 66),   # m 1024: regs 2 / regs 1
    ("cavity", 84, 52),   # m 1025: stream / stream
    ("ogrid", 88, 50),    # m 1032 (odd width): stream with its six colours
    ("ogrid", 90, 49),    # the same width's neighbour: m 1056, an odd number of rows
    ("cavity", 116, 100),  # w 12000: stream
    ("cavity", 117, 100),  # w 12100: stream, far
    ("ogrid", 118, 100),  # w 12100 (odd width): stream, far
]


def _grid(kind, n0, n1):
    return ogrid(n0, n1, ar=1.5, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.1)


def _stencil(g):
    from oracle import oracle
    c = oracle.OracleCase(g, Re=100.0, dt=2e-3)
    return {k: c.field(k) for k in SIP_ORDER}


class Level:
    """The unknowns of a single level: columns 0 .. W-1 when periodic, else 1 .. n0-2; rows 1 .. n1-2."""

    def __init__(self, g, a):
        self.per = g.kind == "ogrid"
        self.W = g.n0 - 1 if self.per else g.n0
        self.a = {k: v[:, :self.W] for k, v in a.items()}
        i, j = np.meshgrid(np.arange(self.W), np.arange(g.n1))
        self.unknown = (j >= 1) & (j <= g.n1 - 2)
        if not self.per:
            self.unknown &= (i >= 1) & (i <= g.n0 - 2)
        colour = (i & 1) | ((j & 1) << 1)
        if self.per and self.W & 1:
            colour = np.where(i == self.W - 1, 4 + (j & 1), colour)
        self.turns = [np.nonzero(self.unknown & (colour == c)) for c in range(colour.max() + 1)]

    def off(self, x, at=None):
        """Sum of the couplings to the neighbours; x is zero outside the unknowns."""
        s = 0.0
        for k, (di, dj) in OFFSETS.items():
            y = np.roll(x, (-dj, -di), (0, 1))
            s = s + (self.a[k] * y if at is None else self.a[k][at] * y[at])
        return s

    def apply(self, x):
        return np.where(self.unknown, self.a["ap"] * x + self.off(x), 0.0)

    def precondition(self, b):
        x = np.zeros_like(b)
        for _ in range(SWEEPS):
            for at in self.turns:
                x[at] = (b[at] - self.off(x, at)) / self.a["ap"][at]
        return x

    def iteration(self, r):
        """The correction after one BiCGStab iteration from residual r."""
        p = self.precondition(r)
        v = self.apply(p)
        alpha = np.sum(r * r) / np.sum(r * v)
        s = r - alpha * v
        z = self.precondition(s)
        t = self.apply(z)
        return alpha * p + np.sum(t * s) / np.sum(t * t) * z


def _close(x, ref):
    assert np.max(np.abs(x - ref)) <= BAR * np.max(np.abs(ref)), np.max(np.abs(x - ref)) / np.max(np.abs(ref))


@pytest.mark.parametrize("kind,n0,n1", GRIDS)
def test_team_kernel(kind, n0, n1):
    g = _grid(kind, n0, n1)
    a = _stencil(g)
    lev = Level(g, a)
    q = np.random.default_rng(n0 * n1).standard_normal((n1, n0))
    rc, phi, iters = sip_gpu(g, [a[k] for k in SIP_ORDER], np.zeros((n1, n0)), q, int(lev.per), tol=0.0, maxit=1)
    assert rc == -5 and iters == 1  # stopped at its cap
    r = np.where(lev.unknown, q[:, :lev.W], 0.0)
    _close(phi[:, :lev.W], lev.iteration(r))


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("kind,n0,n1", GRIDS)
def test_launch_per_phase(kind, n0, n1, mixed):
    from cfd_solver_b200.solver import Batch, case_params
    g = _grid(kind, n0, n1)
    lev = Level(g, _stencil(g))
    p = case_params(g, Re=100.0, Ri=1.0, dt=2e-3, tol_p=0.0, atol_p=0.0, maxit_p=1, precision=mixed)
    with Batch([g], [p]) as b:
        b.profile(True)
        b.step(1)
        assert b.kernel_times()["k_mg_coarse"][1] == 2
        q, pcor = b.plane(0, "q")[:, :lev.W], b.plane(0, "pcor")[:, :lev.W]
        assert b.stats(0)["it_p"] == 1
    x = lev.iteration(np.where(lev.unknown, q, 0.0))
    _close(np.where(lev.unknown, pcor, 0.0), x)
