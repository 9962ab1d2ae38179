"""Frames of many tile rows with few records each have a sorted list, others one built row by row: which of
the two at the rule's lines, the same list either way, and one renderer that goes from one form to the
other and back."""
import numpy as np
import pytest

from helpers import tile_raster_scene

pytestmark = pytest.mark.gpu


def _cams(views, size=(256, 128)):
    from gsr_b200 import scenes

    return [scenes.viewer_camera((7.0 * np.sin(k), 0.5, 7.0 * np.cos(k)), (0.0, 0.0, 0.0), *size, 60.0)
            for k in range(views)]


def _frame(r, cams):
    r.render_views(cams)
    lo, hi, val, ranges, ctl = r.read_back()
    assert ctl.status == 0 and ctl.coverage_mismatch == 0 and ctl.overflow == 0 and ctl.entries > 0
    return (lo, hi, val, ranges, r.read_back_image()), ctl.ext_pad[0] > 0


@pytest.mark.parametrize("count,views,tile,row_wise", [
    (3000, 48, 16, True), (3000, 49, 16, False), (40_000, 49, 16, False), (40_001, 49, 16, True),
    (3000, 24, 8, True), (20_000, 25, 8, False), (20_001, 25, 8, True),
    (3000, 24, 32, True), (65_000, 25, 32, False), (65_001, 25, 32, True)])
def test_the_line(gpu, count, views, tile, row_wise):
    gs = gpu.GpuScene(tile_raster_scene(count, seed=6))
    cams = _cams(views)
    frames = []
    for mode in ("binning", "global"):
        r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, list_mode=mode, tile_size=tile, budget_mb=1024))
        if mode == "global":
            frames.append(_frame(r, cams)[0])
        else:
            for views_now in (2, views, 2, views):  # two views are built row by row
                frame, rows = _frame(r, cams[:views_now])
                assert rows == (row_wise if views_now == views else True)
            frames.append(frame)
        r.close()
    for a, b in zip(*frames):
        np.testing.assert_array_equal(a, b)
    gs.close()


@pytest.mark.parametrize("count,size,views,row_wise", [
    (65_536, (16, 16), 1, True), (65_537, (16, 16), 1, False), (65_537, (17, 16), 1, True),
    (65_536, (32, 300), 1, True), (65_537, (32, 256), 1, True), (65_537, (32, 257), 2, False), (65_537, (33, 257), 1, True)])
def test_single_tiles_and_high_views(gpu, count, size, views, row_wise):
    gs = gpu.GpuScene(tile_raster_scene(count, seed=6))
    frames = []
    for mode in ("binning", "global"):
        r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, list_mode=mode, budget_mb=1024))
        frame, rows = _frame(r, _cams(views, size))
        assert rows == (row_wise and mode == "binning")
        frames.append(frame)
        r.close()
    for a, b in zip(*frames):
        np.testing.assert_array_equal(a, b)
    gs.close()
