"""A case's residual sums do not depend on the batch it is in.

The order in which a sweep's partial residuals are added fixes the last bit of the sum, and with
it the sweep a solve stops at when the tolerance lies next to the residual. The tolerance is put
there by bisection on the case alone (two adjacent doubles, the solve stopping one sweep apart);
beside a case of more than 1024 tiles, whose sums take more threads, both must stop where they
did alone.
"""
import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu


def _params(g, tol, **kw):
    from cfd_solver_b200.solver import case_params
    return case_params(g, **dict(dict(Re=250.0, Ri=1.0, dt=2e-3 if g.kind == "cavity" else 1e-3, tol_mom=tol,
                                      atol_mom=0.0), **kw))


def _image(b):
    img = np.zeros(b.state_bytes() // 8)
    b.get_state(img)
    return img


@pytest.mark.parametrize("make,field", [(lambda: cavity(289, 289, skew=0.1), 0), (lambda: cavity(289, 289, skew=0.1), 2),
                                        (lambda: ogrid(321, 257, skew=0.1), 1)])
def test_stop_decisions_alone_and_beside_a_large_case(make, field):
    from cfd_solver_b200.solver import Batch
    g, large = make(), cavity(1025, 1025, skew=0.1)
    with Batch([g], [_params(g, 1e-3)]) as b:
        b.step(3)
        start = _image(b)

    def alone(tol):
        with Batch([g], [_params(g, tol)]) as b:
            b.set_state(start)
            b.step(1)
            return b.stats(0)["it_mom"]

    # the first tolerance below 1e-2 at which the field's solve stops a sweep later
    hi = 1e-2
    lo, at_hi = hi, alone(hi)[field]
    while alone(lo)[field] == at_hi:
        lo *= 0.5
    lo, hi = np.float64(lo), np.float64(hi)
    while np.nextafter(lo, 1.0) < hi:
        mid = np.int64((lo.view(np.int64) + hi.view(np.int64)) // 2).view(np.float64)
        lo, hi = (lo, mid) if alone(mid)[field] == at_hi else (mid, hi)
    expect = {tol: alone(tol) for tol in (lo, hi)}
    assert expect[lo][field] > expect[hi][field]
    with Batch([large, g], [_params(large, 1e-2, Re=1000.0), _params(g, 1e-2)]) as b:
        both = _image(b)
        both[-start.size:] = start
        for tol in (lo, hi):
            b.admit(1, g, _params(g, tol))
            b.set_state(both)
            b.step(1)
            assert b.stats(1)["it_mom"] == expect[tol], (tol, expect)
