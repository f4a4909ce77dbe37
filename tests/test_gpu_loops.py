"""The step graph of a batch too large for the team kernel: its chained launches and its loops.

160 cases do not fit as teams, so they run as the step graph, whose kernels begin while the one
before drains and whose momentum loop holds several sweeps per iteration. The host-driven step
(per-launch profiling) launches one kernel after another, and the same case alone runs in the
team kernel: all three must give the same bits, and a solve that cannot converge must stop after
exactly the sweeps its cap allows (an even number in the FP64 form), at every remainder of the
cap by the loop body.
"""
import numpy as np
import pytest

from cfd_solver_b200 import _lib
from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu


def _run(grids, params, host):
    from cfd_solver_b200.solver import Batch
    with Batch(grids, params) as b:
        b.profile(host)
        b.step(3)
        img = np.zeros(b.state_bytes() // 8)
        b.get_state(img)
        return img.view(np.int64), {k: b.plane(0, k) for k in ("u", "v", "T", "p", "q")}, b.all_stats()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("maxit", [2, 3, 4, 5, 6, 7, 9, 100])
def test_graph_host_and_team_agree_at_every_cap(mixed, maxit):
    from cfd_solver_b200.solver import case_params
    grids = [ogrid(33 + 2 * (k % 3), 21, skew=0.1) if k % 2 else cavity(40, 26 + k % 5, skew=0.1) for k in range(160)]
    prec = _lib.PRECISION_MIXED if mixed else _lib.PRECISION_FP64
    tol = 1e-7 if maxit == 100 else 0.0  # 0: no solve converges, all stop at the cap
    params = [case_params(g, Re=150.0, Ri=0.5, Pr=0.71, dt=1e-3, precision=prec, tol_mom=tol, atol_mom=0.0,
                          maxit_mom=maxit) for g in grids]
    a, fa, sa = _run(grids, params, False)
    h, fh, sh = _run(grids, params, True)
    np.testing.assert_array_equal(a, h)
    assert sa == sh
    _, ft, st = _run(grids[:1], params[:1], False)
    for k in fa:
        np.testing.assert_array_equal(fa[k].view(np.int64), ft[k].view(np.int64), err_msg=k)
    assert sa[0]["it_mom"] == st[0]["it_mom"]
    if maxit < 100:
        cap = maxit if mixed else maxit // 2 * 2
        assert all(list(s["it_mom"])[0] == cap and s["status"] & 1 for s in sa), (sa[0]["it_mom"], cap)
    else:
        assert all(max(s["it_mom"]) < 100 and not s["status"] & 1 for s in sa)
