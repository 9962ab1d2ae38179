"""The binning list built row by row (rows of tiles as buckets, then the tiles of a row) against the
global mode's sorted list, entry for entry, over the forms it accepts: every bounds mode and record
format, all three tile shapes, runs of one row and splats of many rows (spilled runs, more of them than
the spill holds), one gaussian and frames of several small views, image sides at its limits (256 tile
rows, 512 tiles a row) and one past them, where the list is sorted. Over its capacity the list is the
full one cut in (view, depth, gaussian, tile) order."""
import numpy as np
import pytest

from helpers import tile_raster_scene

pytestmark = pytest.mark.gpu


def _frames(gpu, gs, cams, **kw):
    out = []
    for mode in ("binning", "global"):
        r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, list_mode=mode, **kw))
        r.render_views(cams)
        ctl = r.read_control()
        assert ctl.status == 0 and ctl.coverage_mismatch == 0, ctl.as_dict()
        out.append((r.read_back(), r.read_back_image(), ctl))
        r.close()
    return out


def _equal(rows, glob):
    for a, b in zip(rows[0][:4], glob[0][:4]):
        np.testing.assert_array_equal(a, b)
    assert rows[1].tobytes() == glob[1].tobytes()
    for k in ("visible", "duplicates", "entries", "overflow", "tile_max"):
        assert getattr(rows[2], k) == getattr(glob[2], k), k


def _cam(w, h, fovy=60.0, eye=(0.3, 0.5, 6.0)):
    from gsr_b200 import scenes

    return scenes.viewer_camera(eye, (0.0, 0.0, 0.0), w, h, fovy)


@pytest.mark.parametrize("size,tile,row_wise", [((16, 4096), 16, True), ((16, 4097), 16, False), ((8192, 24), 16, True),
                                                ((8193, 24), 16, False), ((40, 2048), 8, True), ((40, 2049), 8, False),
                                                ((64, 2040), 32, True), ((1, 1), 16, True), ((1000, 700), 8, True)])
def test_image_sides(gpu, size, tile, row_wise):
    gs = gpu.GpuScene(tile_raster_scene(5000, seed=5, needles=True))
    rows, glob = _frames(gpu, gs, [_cam(*size)], tile_size=tile)
    _equal(rows, glob)
    assert (rows[2].ext_pad[0] > 0) == (row_wise and rows[2].entries > 0)


@pytest.mark.parametrize("bounds", ["tight", "rect", "cutoff-only"])
@pytest.mark.parametrize("splat", ["full", "p32", "p24"])
@pytest.mark.parametrize("count", [1, 33, 4000])
def test_forms(gpu, bounds, splat, count):
    gs = gpu.GpuScene(tile_raster_scene(count, seed=9, needles=True))
    _equal(*_frames(gpu, gs, [_cam(650, 390)], bounds=bounds, render_splat=splat))


@pytest.mark.parametrize("count", [300, 40_000])
def test_tall_splats_spill(gpu, count):
    """Vertical needles over all 68 tile rows: 300 fill a block's own part of the spilled runs, 40,000
    need 2.7 M runs where the frame has 0.2 M, so most are computed again from their ellipses."""
    scene = tile_raster_scene(count, seed=3)
    n = np.arange(count)
    scene.pos_alpha[:, :3] = np.stack([(n % 997) / 997.0 * 9.0 - 4.5, np.zeros(count), (n % 31) * 0.01], 1)
    scene.pos_alpha[:, 3] = 0.5
    scene.scales[:, :3] = (0.002, 3.0, 0.002)
    scene.rotations[:] = (1.0, 0.0, 0.0, 0.0)
    gs = gpu.GpuScene(scene)
    rows, glob = _frames(gpu, gs, [_cam(1920, 1080)], budget_mb=512)
    assert rows[2].entries > 60 * count
    _equal(rows, glob)


@pytest.mark.parametrize("count", [1, 700, 3000])
def test_small_views(gpu, count):
    from gsr_b200 import scenes

    gs = gpu.GpuScene(scenes.make_scene(count, seed=count, ball_radius=3.0))
    cams = [_cam(w, h, eye=(4.0 * np.sin(k), 0.5, 4.0 * np.cos(k)))
            for k, (w, h) in enumerate([(16, 16), (333, 100), (17, 250), (640, 8), (256, 256), (100, 333)])]
    _equal(*_frames(gpu, gs, cams))


@pytest.mark.parametrize("views", [1, 3])
@pytest.mark.parametrize("budget_mb", [1, 2])
def test_overflow_cuts_in_depth_order(gpu, views, budget_mb):
    scene = tile_raster_scene(90_000, seed=17, needles=True)
    gs = gpu.GpuScene(scene)
    cams = [_cam(640, 360, eye=(0.3 + k, 0.5, 6.0)) for k in range(views)]
    full = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, budget_mb=512, list_mode="global"))
    full.render_views(cams)
    lo, hi, val, _, fctl = full.read_back()
    layouts = full.view_layouts()
    r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, budget_mb=budget_mb))
    for _ in range(2):  # the second frame reuses every buffer
        r.render_views(cams)
    glo, ghi, gval, ranges, ctl = r.read_back()
    cap = r.capacity()[0]
    assert ctl.status == 0 and ctl.entries == cap and ctl.duplicates == fctl.duplicates
    assert ctl.overflow == fctl.duplicates - cap
    view = np.searchsorted([v.tile_base for v in layouts], hi, side="right")
    keep = np.lexsort((hi, val, lo, view))[:cap]
    keep = keep[np.lexsort((val[keep], lo[keep], hi[keep]))]
    np.testing.assert_array_equal(ghi, hi[keep])
    np.testing.assert_array_equal(glo, lo[keep])
    np.testing.assert_array_equal(gval, val[keep])
    counts = np.bincount(ghi, minlength=len(ranges))
    np.testing.assert_array_equal(ranges[:, 1] - ranges[:, 0], counts)
    r.close()
    full.close()


def test_forced_timeout_is_reported_and_recoverable(gpu):
    gs = gpu.GpuScene(tile_raster_scene(50_000, seed=2))
    r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False))
    cams = [_cam(640, 360), _cam(320, 240)]
    r.render_views(cams)
    good = r.read_back()
    r.force_timeout(2000)
    r.render_views(cams)
    assert r.read_control().status & gpu.CONTROL_TIMEOUT
    r.render_views(cams)
    again = r.read_back()
    assert again[4].status == 0
    for a, b in zip(good[:4], again[:4]):
        np.testing.assert_array_equal(a, b)
    r.close()
