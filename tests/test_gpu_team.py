"""The team kernel (whole steps of a case in one launch) against the launch-per-phase step.

Both evaluate the same expressions and sum in the same order, so a batch small enough for teams
must give the bits of the host-driven step (per-launch profiling always takes that path), in
every field and statistic, at the sizes where the team kernel's forms change: clusters and
shares of a cooperative grid, one warp or a block for the totals, levels run by one CTA, one
or two points of a colour per thread on the coarsest level or none of it in registers, an
empty slot, a solve stopped at its cap, a moving wall.
"""
import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "T", "p", "up", "vp", "pcor", "q", "vort", "dil")


def _run(grids, params, host, chunks=(1, 2, 4), empty=None):
    from cfd_solver_b200.solver import Batch
    with Batch(grids, params) as b:
        if empty is not None:
            b.set_active(empty, False)
        b.profile(host)
        n0 = b.launches()
        for n in chunks:
            b.step(n)
        n1 = b.launches()
        img = np.zeros(b.state_bytes() // 8)
        b.get_state(img)
        out = [{k: b.plane(c, k) for k in FIELDS} for c in range(min(len(grids), 3))]
        return img.view(np.int64), out, b.all_stats(), n1 - n0


def _same(grids, params, team=True, **kw):
    a, fa, sa, la = _run(grids, params, False, **kw)
    b, fb, sb, lb = _run(grids, params, True, **kw)
    # one launch per call, and per 32 steps of it
    assert (la == sum(-(-n // 32) for n in kw.get("chunks", (1, 2, 4)))) == team, la
    np.testing.assert_array_equal(a, b)
    for x, y in zip(fa, fb):
        for k in x:
            np.testing.assert_array_equal(x[k].view(np.int64), y[k].view(np.int64), err_msg=k)
    for x, y in zip(sa, sb):
        assert x == y or x["status"] & 4, (x, y)
    return sa


def _case(kind, n0, n1, mixed=False, dt=None, **kw):
    from cfd_solver_b200 import _lib
    from cfd_solver_b200.solver import case_params
    g = ogrid(n0, n1, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.12)
    prec = _lib.PRECISION_MIXED if mixed else _lib.PRECISION_FP64
    p = dict(Re=250.0, Ri=1.0, Pr=0.71, dt=dt or (1e-4 if kind == "ogrid" else 2e-3), precision=prec)
    return g, case_params(g, **dict(p, **kw))


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kind,n0,n1", [
    ("ogrid", 8, 6), ("cavity", 8, 8),        # the smallest grids: one tile, one level
    ("ogrid", 33, 19), ("cavity", 34, 18),    # one tile more than a row of 32 x 16
    ("ogrid", 65, 65), ("cavity", 65, 65),    # clusters; the lower levels in one CTA
    ("ogrid", 129, 131), ("cavity", 131, 129),  # 33 and 40 tiles: a block sums the totals
    ("ogrid", 46, 46),    # odd width, one level: six colours
    ("ogrid", 181, 91),   # coarsest level 90 x 44: two points of a colour per thread
    ("ogrid", 131, 130),  # coarsest level 65 x 128 by one CTA: stencils re-read in every pass
    ("cavity", 257, 193),  # a share of the grid: 96 tiles
])
def test_single_case_equals_host_driven(kind, n0, n1, mixed):
    g, p = _case(kind, n0, n1, mixed)
    _same([g], [p])


@pytest.mark.parametrize("n,kind,n0,n1,team", [
    (17, "ogrid", 33, 25, True), (40, "ogrid", 33, 33, True), (148, "ogrid", 17, 17, True),
    (149, "ogrid", 17, 17, False),            # more cases than SMs: the step graph
    (5, "cavity", 129, 97, True), (16, "ogrid", 129, 129, True), (30, "cavity", 129, 129, True),
    (38, "cavity", 129, 129, False),          # more than 8 tiles per CTA of teams of up to 4
    (2, "cavity", 385, 385, True), (2, "ogrid", 417, 417, False),     # 4 / 5 per CTA of teams of 74
    (10, "ogrid", 193, 193, True), (16, "ogrid", 193, 193, False),   # 6 / 8 per CTA of teams of 14 / 9
])
def test_batches_around_the_rule(n, kind, n0, n1, team):
    made = [_case(kind, n0, n1, Re=100.0 + 7 * k) for k in range(n)]
    _same([g for g, _ in made], [p for _, p in made], team=team, chunks=(1, 2))


def test_mixed_sizes_and_an_empty_slot():
    made = [_case("ogrid", 65, 49), _case("cavity", 41, 33), _case("ogrid", 97, 65), _case("cavity", 66, 35)]
    st = _same([g for g, _ in made], [p for _, p in made], empty=2)
    assert st[2]["steps"] == 0 and st[1]["steps"] == 7


def test_statuses_and_moving_wall():
    g, p = _case("ogrid", 65, 49, tol_p=1e-15, maxit_p=3, tol_mom=1e-15, maxit_mom=5)
    assert _same([g], [p])[0]["status"] & 1
    g, p = _case("ogrid", 65, 49, F=0.7, time_accurate=1, dt=1e-2)
    _same([g], [p], chunks=(3, 40))
    g, p = _case("cavity", 65, 65, mixed=True, tol_mom=1e-9, maxit_mom=7)
    _same([g], [p])


def test_graph_and_team_steps_mix():
    """A schedule only the launch-per-phase step has, between team steps of the same batch."""
    from cfd_solver_b200.solver import Batch
    g, p = _case("ogrid", 65, 65)
    out = []
    for host in (False, True):
        with Batch([g], [p]) as b:
            b.profile(host)
            b.step(3)
            b.set_mg(1, 3, 12, 1)
            b.step(3)
            b.set_mg(1, 3, 12, 2)
            b.step(3)
            out.append((b.plane(0, "p"), b.stats(0)))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
