"""The state image is packed and unpacked in row blocks of 16: every size of a last block, rows
narrower and wider than a warp, both grid profiles, cases of different heights in one image.
Copies only, so everything is equal to the bit.
"""
import numpy as np
import pytest

from cfd_solver_b200.grid import cavity, ogrid

pytestmark = pytest.mark.gpu

PLANES = ("u", "v", "p", "T", "up", "vp")  # the image's order


def _grid(kind, n0, n1):
    return ogrid(n0, n1, skew=0.1) if kind == "ogrid" else cavity(n0, n1, skew=0.1)


@pytest.mark.parametrize("cases", [
    [("cavity", 9, 15)], [("cavity", 33, 16)], [("ogrid", 34, 17)], [("ogrid", 131, 32)], [("cavity", 160, 33)],
    [("ogrid", 34, 17), ("cavity", 70, 9), ("ogrid", 41, 130), ("cavity", 33, 48)],
])
def test_image_holds_the_planes_and_comes_back(cases):
    from cfd_solver_b200.solver import Batch, case_params
    grids = [_grid(*c) for c in cases]
    params = [case_params(g, Re=120.0, Ri=0.5, Pr=0.71, dt=1e-3) for g in grids]
    with Batch(grids, params) as a, Batch(grids, params) as b:
        a.step(3)
        img = np.full(a.state_bytes() // 8, np.nan)
        a.get_state(img)
        o = 0
        for k, (kind, n0, n1) in enumerate(cases):
            nc = n0 - (kind == "ogrid")  # stored columns
            for name in PLANES:
                np.testing.assert_array_equal(img[o:o + n1 * nc].reshape(n1, nc), a.plane(k, name)[:, :nc], err_msg=name)
                o += n1 * nc
            assert list(img[o:o + 1].view(np.int32)) [1] == 3  # steps taken
            o += 16
        assert o == img.size
        b.set_state(img)
        a.step(2)
        b.step(2)
        back = [np.zeros_like(img), np.zeros_like(img)]
        a.get_state(back[0])
        b.get_state(back[1])
        np.testing.assert_array_equal(back[0].view(np.int64), back[1].view(np.int64))
