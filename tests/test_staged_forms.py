"""What chooses the form of the staged back-projection (host only): mr_staged_traits against the
tiles and footprints counted in NumPy, and the launches that go to the four-warp form."""
import ctypes

import numpy as np
import pytest

from tomography_local_demo_b200 import _native as N
from tomography_local_demo_b200 import circular_cone_vectors
from tomography_local_demo_b200 import recon as R

ROWS, COLS, VIEWS = 384, 486, 600
GEOM = circular_cone_vectors(VIEWS, 440.0, 680.0, ROWS, COLS, 145.3 / COLS)
MAPS = R.cone_view_maps(R.cone_constants(GEOM.vectors), ROWS, COLS)
PIXEL = 145.3 / COLS * 440.0 / 680.0


def traits(grid, dtype=N.MR_F32):
    return R.staged_traits(MAPS, N.MR_CONE, ROWS, COLS, dtype, grid.tobytes())


def plane(normal, n, zoom=1.0, origin=(0.0, 0.0, 0.5)):
    return R.plane_grid(GEOM.volume_box(), origin, normal, n, None, zoom)


@pytest.mark.parametrize("normal", [(0.0, 0.0, 1.0), (0.0, 1.0, 0.0), (0.5, 0.4, 0.7), (-0.1, 0.3, 0.9)])
@pytest.mark.parametrize("n,zoom", [(31, 1.0), (33, 0.3), (200, 1.0), (401, 0.25), (257, 4.0)])
def test_busy_tiles(normal, n, zoom):
    g = plane(normal, n, zoom, tuple(3.0 * np.asarray(normal)))
    a = (np.arange(n) - g["mask_half"]) * g["mask_delta"]
    p = g["mask_c"] + a[None, :, None] * g["mask_ej"] + a[:, None, None] * g["mask_ei"]
    inside = (np.abs(p) <= g["box"]).all(-1)
    exact = sum(inside[i:i + 32, j:j + 32].any() for i in range(0, n, 32) for j in range(0, n, 32))
    # a tile that only reaches past one face near a corner of the box counts too: never fewer
    # than exact, and at most the tiles within one tile of a busy one
    near = sum(inside[max(0, i - 32):i + 64, max(0, j - 32):j + 64].any() for i in range(0, n, 32) for j in range(0, n, 32))
    assert exact <= traits(g)[0] <= near


@pytest.mark.parametrize("dtype", [N.MR_F32, N.MR_BF16, N.MR_F16])
def test_shares(dtype):
    def shares(normal, pixels):                    # a slice of 192 samples a side at that many pixels a sample
        size = 192 * pixels * PIXEL
        return traits(R.plane_grid(3 * GEOM.volume_box(), (0, 0, 0.5), normal, 192, size), dtype)[1:]
    assert shares((0, 0, 1.0), 1.0) == (1.0, 0.0)
    assert shares((0, 1.0, 0), 1.0) == (1.0, 0.0)
    staged, wide = shares((0, 0, 1.0), 3.0)
    assert staged + wide == 1.0 and wide > 0.9     # the few others lie off the detector
    assert shares((0, 1.0, 0), 4.0)[1] == 0.0      # as tall as wide: in no box
    assert shares((0, 0, 1.0), 14.0)[1] == 0.0     # wider than any box


def test_launches_of_the_four_warp_form():
    pays = N.load().mr_staged_slim_pays
    # a wave is 104 clusters of the full form, 142 (FP32) or 175 of the four-warp one: neither
    # inside the full form's first wave nor just past the end of one of its own
    assert [pays(n, N.MR_F32) for n in (0, 64, 104, 128, 147, 256, 288, 400, 3600)] == [0, 0, 0, 1, 0, 1, 0, 1, 1]
    assert [pays(n, N.MR_BF16) for n in (0, 64, 104, 128, 180, 256, 400, 768, 3600)] == [0, 0, 0, 1, 0, 1, 1, 1, 1]
    small, large = plane((0.5, 0.4, 0.7), 128), plane((0.5, 0.4, 0.7), 512)
    full = plane((0, 0, 1.0), 1024)
    for dtype in (N.MR_F32, N.MR_BF16):
        assert R.slim_pays([traits(full, dtype)], dtype)
        assert R.slim_pays([traits(large, dtype)] * 3, dtype)
        assert not R.slim_pays([traits(large, dtype), traits(small, dtype)], dtype)      # 4.5 pixels a sample: not staged
        # 1024 tiles, 42 of them in the box
        assert not R.slim_pays([traits(plane((0.5, 0.4, 0.7), 1024, 0.25), dtype)], dtype)
        assert not R.slim_pays([], dtype)
    # some grids that are staged in part, in a list of many tiles and in a shorter one
    part, whole = (300, 0.5, 0.0), (300, 1.0, 0.0)
    assert [R.slim_pays([part] * a + [whole] * b, N.MR_BF16) for a, b in ((1, 2), (2, 6), (5, 3))] == [False, True, False]
    assert [R.slim_pays([(60, 0.7, 0.0)] + [whole] * b, N.MR_F32) for b in (3, 9, 10)] == [False, False, True]
    assert R.slim_grids([whole, part], N.MR_F32) is False and R.slim_grids([whole] * 2, N.MR_F32) is True
    assert R.slim_grids([part] * 3 + [(6000, 1.0, 0.0)], N.MR_F32) == [False] * 3 + [True]


@pytest.mark.parametrize("dtype", [N.MR_F32, N.MR_BF16])
def test_only_footprints_that_wide_boxes_hold_are_wide(dtype):
    def chosen(normal, pixels, count, n=192):
        grids = [R.plane_grid(3 * GEOM.volume_box(), (0, 0, 0.5), normal, n, n * pixels * PIXEL)] * count
        wide = [R.is_wide(g, (0.0, 0.0, 1.0), R.WIDE_TILE_PIXELS / 31 * PIXEL) for g in grids]
        assert wide == [True] * count
        return R.wide_grids(wide, [traits(g, dtype) for g in grids])
    assert chosen((0, 0, 1.0), 2.6, 25) == [True] * 25           # trial slices of a rotation-centre search
    assert chosen((0, 0, 1.0), 2.6, 1) == [True]
    assert chosen((0, 1.0, 0), 3.0, 25) == [False] * 25          # as tall as wide
    assert chosen((0.5, 0.4, 0.7), 3.0, 25) == [False] * 25
    assert chosen((0, 0, 1.0), 14.0, 25, 64) == [False] * 25     # 434 columns
    # 186 to 263 columns: a part of the views is in a box, which one slice's tiles do not wait for
    assert chosen((0, 0, 1.0), 6.0, 25, 96) == [True] * 25
    assert chosen((0, 0, 1.0), 6.0, 1, 96) == [False]


@pytest.mark.parametrize("dtype", [N.MR_F32, N.MR_BF16])
def test_few_wide_tiles_share_the_launch_of_the_others(dtype):
    axial = R.plane_grid(GEOM.volume_box(), (0, 0, 0.5), (0, 0, 1.0), 192)               # 36 tiles
    other = plane((0.5, 0.4, 0.7), 128)
    ta, to = traits(axial, dtype), traits(other, dtype)
    for count in (1, 3, 11):
        assert R.wide_grids([True] * count + [False], [ta] * count + [to]) == [False] * (count + 1)
        assert R.wide_grids([True] * count, [ta] * count) == [True] * count
    assert R.wide_grids([True] * 12 + [False], [ta] * 12 + [to]) == [True] * 12 + [False]


def test_traits_argument_checks():
    lib, t = N.load(), (ctypes.c_double * 3)()
    ok = [MAPS.ctypes.data, VIEWS, N.MR_CONE, ROWS, COLS, N.MR_F32, plane((0, 0, 1.0), 64).tobytes(), t]
    assert lib.mr_staged_traits(*ok) == 0
    for at, bad in ((0, None), (1, 0), (2, 7), (3, 0), (4, -1), (5, 9), (6, None), (7, None)):
        assert lib.mr_staged_traits(*(ok[:at] + [bad] + ok[at + 1:])) == N.MR_ERR_INVALID
    points = plane((0, 0, 1.0), 64)
    points["flags"] = N.MR_GRID_POINTS
    assert lib.mr_staged_traits(*(ok[:6] + [points.tobytes(), t])) == N.MR_ERR_INVALID


@pytest.mark.parametrize("dtype", [N.MR_F32, N.MR_BF16, N.MR_F16])
def test_both_wide_boxes_occur_where_they_are_compared(dtype):
    """The geometry of test_wide_boxes_change_nothing: tilted slices whose footprints are too tall
    for FP32's wider box, axial ones that are too wide for the narrower box."""
    from oracle import geometry as og
    maps = R.cone_view_maps(R.cone_constants(og.circular_cone_vectors(29, 440.0, 680.0, 0.3)), 90, 420)
    pixel, box = 0.3 * 440.0 / 680.0, np.array([40.0, 40.0, 9.0])

    def wide(normal, pitch):
        grid = R.plane_grid(box, (1.0, 2.0, 0.4), normal, 45, 45 * pitch * pixel)
        return R.staged_traits(maps, N.MR_CONE, 90, 420, dtype, grid.tobytes())[2]
    assert wide((0.1, -0.05, 1.0), 4.2) > 0.5                            # 130 to 184 columns, 20 rows
    assert wide((0.0, 0.0, 1.0), 5.5) > 0.3                              # 170 to 241 columns: the wider box
