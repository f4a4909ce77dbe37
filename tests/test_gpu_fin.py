"""The per-case totals at the edges of their sums.

The tile kernels write one partial row per tile and k_fin adds a case's rows with 256 threads, so
the tile counts here are one row, one pass of the threads less, exactly and two more, and a
case after others in the same tables. The totals must be those of the fields themselves. Each
sum of n nonnegative terms in double is within n 2^-53 of the exact one, relatively, so two
orders differ by at most 2 n 2^-53; the maxima are exact.
"""
import numpy as np
import pytest

from cfd_solver_b200.grid import cavity

pytestmark = pytest.mark.gpu

# cavities of a x b tiles of 32 x 16 unknowns: 1, 255, 256, 258 tiles, and a ragged edge
SIZES = [(34, 18), (17 * 32 + 2, 15 * 16 + 2), (16 * 32 + 2, 16 * 16 + 2), (43 * 32 + 2, 6 * 16 + 2), (41, 31)]


@pytest.mark.parametrize("picked", [[k] for k in range(len(SIZES))] + [[4, 1, 0, 3, 2]])
def test_totals_are_those_of_the_fields(picked):
    from cfd_solver_b200.solver import Batch, case_params
    grids = [cavity(*SIZES[k], skew=0.1) for k in picked]
    dt = 1e-3
    params = [case_params(g, Re=100.0, Ri=0.5, Pr=0.71, dt=dt) for g in grids]
    with Batch(grids, params) as b:
        b.profile(True)  # always the launch-per-phase step
        b.step(1)
        before = [{f: b.plane(c, f) for f in ("u", "v", "T")} for c in range(len(grids))]
        b.step(1)
        for c, g in enumerate(grids):
            n1, n0 = before[c]["u"].shape
            n = (n0 - 2) * (n1 - 2)
            tol = 2 * n * 2.0 ** -53
            s = b.all_stats()[c]
            d = {f: np.abs(b.plane(c, f) - before[c][f])[1:-1, 1:-1] for f in before[c]}
            q = b.plane(c, "q")[1:-1, 1:-1]
            assert s["dT_max"] == d["T"].max()
            assert s["dT_l1"] == pytest.approx(d["T"].sum(), rel=tol, abs=0)
            assert s["q_max"] == np.abs(q).max()
            assert s["q_l1"] == pytest.approx(np.abs(q).sum(), rel=tol, abs=0)
            assert s["q_l2"] == pytest.approx(np.sqrt((q * q).sum()), rel=tol, abs=0)
            # |du| + |dv| are added per cell first: two more roundings, and the division
            sr = (d["u"].sum() + d["v"].sum() + d["T"].sum()) / (dt * n)
            assert s["steady_res"] == pytest.approx(sr, rel=2 * tol + 8 * 2.0 ** -53, abs=0)
