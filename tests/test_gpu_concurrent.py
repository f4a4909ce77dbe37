"""Several batches stepped at once by threads of one process.

Team launches that together ask for more SMs than the chip has take turns, so such batches step by
the graph, whose launches overlap; batches whose teams fit side by side stay with one launch per
call. Whatever the route, every batch has the bits it has alone.
"""
import threading

import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu


def _batch(kind, n0, n1, n, k):
    from cfd_solver_b200.solver import Batch, case_params
    g = ogrid(n0, n1, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.1)
    p = case_params(g, Re=150.0 + 10 * k, Ri=1.0, dt=1e-4 if kind == "ogrid" else 2e-3)
    return Batch([g] * n, [p] * n)


def _image(b):
    img = np.zeros(b.state_bytes() // 8)
    b.get_state(img)
    return img.view(np.int64)


def _together(batches, calls):
    """Every batch steps through its list of calls in a thread of its own; exceptions are passed on."""
    start, errors = threading.Barrier(len(batches)), []

    def work(b, c):
        try:
            start.wait(60)
            for n in c:
                b.step(n)
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=a) for a in zip(batches, calls)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("kind,n0,n1,n,k,team", [
    ("ogrid", 257, 257, 1, 2, False),  # two teams of the whole chip
    ("cavity", 129, 129, 4, 5, False),  # five batches of four clusters of 16
    ("ogrid", 65, 65, 1, 4, True),     # four clusters of 16 side by side
    ("ogrid", 65, 65, 2, 10, True),    # ten batches of two clusters of 16: a quarter of the chip each at most
])
@pytest.mark.parametrize("calls", [[1] * 200, [100, 100]])
def test_batches_stepped_at_once(kind, n0, n1, n, k, team, calls):
    batches = [_batch(kind, n0, n1, n, j) for j in range(k)]
    try:
        _together(batches, [calls] * k)
        launches = [b.launches() for b in batches]
        images = [_image(b) for b in batches]
    finally:
        for b in batches:
            b.close()
    for j in range(k):
        with _batch(kind, n0, n1, n, j) as b:
            for m in calls:
                b.step(m)
            alone = b.launches()
            np.testing.assert_array_equal(_image(b), images[j], err_msg=str(j))
        if team:
            assert launches[j] == alone
        else:  # most of the 200 steps went launch by launch (some 30 launches a step)
            assert launches[j] > alone + 100 * 20, (launches[j], alone)


def test_small_steps_beside_a_large_team():
    """A team that holds the chip gives way to a small batch's calls, which would wait for it."""
    calls = [[100] * 6, [1] * 300]
    pair = [_batch("ogrid", 257, 257, 1, 0), _batch("ogrid", 65, 65, 1, 1)]
    try:
        _together(pair, calls)
        launches, images = [b.launches() for b in pair], [_image(b) for b in pair]
    finally:
        for b in pair:
            b.close()
    for j, (n, kind) in enumerate(((257, "ogrid"), (65, "ogrid"))):
        with _batch(kind, n, n, 1, j) as b:
            for m in calls[j]:
                b.step(m)
            alone = b.launches()
            np.testing.assert_array_equal(_image(b), images[j], err_msg=str(j))
        assert launches[j] > alone + 64 * 20 if j == 0 else launches[j] == alone, (launches[j], alone)
