"""Steps whose pressure solve has nothing to do, by the team kernel and launch by launch.

A continuity source that sums to zero (a cavity at rest) or to something not finite (a NaN planted
in `up` alone, so that u and v are still finite when the solve would start) ends the solve
before its first barrier. Every CTA of a team must have read the source's partial sums before the
correction's are stored, or CTAs could disagree about the solve. Same fields, statistics and
status words as the host-driven step, in clusters and in a share of the grid.
"""
import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "T", "p", "up", "vp", "pcor", "q", "vort", "dil")
PLANES = 6  # of the state image: u, v, p, T, up, vp


def _grids(kind, n0, n1, n):
    from cfd_solver_b200.solver import case_params
    g = ogrid(n0, n1, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.12)
    return g, (lambda **kw: [case_params(g, **dict(dict(Re=250.0, dt=1e-4 if kind == "ogrid" else 2e-3), **kw))] * n)


def _run(grids, params, host, plant=None, steps=(1, 3)):
    from cfd_solver_b200.solver import Batch
    with Batch(grids, params) as b:
        if plant is not None:
            b.step(2)
            img = np.zeros(b.state_bytes() // 8)
            b.get_state(img)
            g = grids[plant]
            w = g.n0 - 1 if g.kind == "ogrid" else g.n0
            img[plant * (PLANES * g.n1 * w + 16) + (4 * g.n1 + g.n1 // 2) * w + w // 2] = np.nan
            b.set_state(img)
        b.profile(host)
        n0 = b.launches()
        for n in steps:
            b.step(n)
        launches = b.launches() - n0
        out = [{k: b.plane(c, k) for k in FIELDS} for c in range(len(grids))]
        return out, b.all_stats(), launches


def _same(x, y):
    for fx, fy in zip(x[0], y[0]):
        for k in FIELDS:
            np.testing.assert_array_equal(fx[k], fy[k], err_msg=k)  # NaN equals NaN
    for sx, sy in zip(x[1], y[1]):
        for k in sx:
            np.testing.assert_array_equal(sx[k], sy[k], err_msg=k)


# clusters of 16 and of 8 CTAs; shares of 148 and of 74 CTAs of the grid
SIZES = [(65, 65, 1), (65, 65, 12), (257, 193, 1), (257, 257, 2)]


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("n0,n1,n", SIZES)
def test_case_at_rest(n0, n1, n, mixed):
    g, params = _grids("cavity", n0, n1, n)
    ps = params(lid_u=0.0, Ri=0.0, precision=mixed)
    a, b = _run([g] * n, ps, False), _run([g] * n, ps, True)
    assert a[2] == 2  # one launch per call: the team kernel
    _same(a, b)
    for s in a[1]:
        assert s["it_p"] == 0 and s["status"] == 0
    assert not np.any(a[0][0]["u"]) and np.any(a[0][0]["T"])


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("kind", ["ogrid", "cavity"])
@pytest.mark.parametrize("n0,n1,n", SIZES)
def test_nan_in_up_alone(kind, n0, n1, n, mixed):
    g, params = _grids(kind, n0, n1, n)
    ps = params(warm_start=1, precision=mixed)
    bad = n - 1
    a, b = _run([g] * n, ps, False, plant=bad, steps=(1,)), _run([g] * n, ps, True, plant=bad, steps=(1,))
    assert a[2] == 1
    _same(a, b)
    assert a[1][bad]["status"] & 4 and a[1][bad]["it_p"] == 0
    for s in a[1][:bad]:
        assert s["status"] == 0 and s["it_p"] > 0
