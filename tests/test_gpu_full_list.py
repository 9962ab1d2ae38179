"""Row-wise lists that are full long before the frame's last record: the cut in the first block of records,
in the first view of several, and in a later one. The list is the global mode's cut at its capacity in
(view, depth, gaussian, tile) order, in repeated frames."""
import numpy as np
import pytest

from helpers import tile_raster_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bounds", ["rect", "tight"])
@pytest.mark.parametrize("count,scale,views", [(3000, 20.0, 1), (3000, 20.0, 5), (40_000, 1.0, 5), (200_000, 0.2, 3)])
def test_cut_before_the_end(gpu, count, scale, views, bounds):
    from gsr_b200 import scenes

    scene = tile_raster_scene(count, seed=count)
    scene.scales[:] *= np.float32(scale)
    gs = gpu.GpuScene(scene)
    cams = [scenes.viewer_camera((0.3 + k, 0.5, 6.0), (0.0, 0.0, 0.0), 640, 360, 60.0) for k in range(views)]
    full = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, budget_mb=2048, list_mode="global", bounds=bounds))
    full.render_views(cams)
    lo, hi, val, _, fctl = full.read_back()
    assert fctl.status == 0 and fctl.overflow == 0
    view = np.searchsorted([v.tile_base for v in full.view_layouts()], hi, side="right")
    full.close()
    r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, budget_mb=1, bounds=bounds))
    order = None
    for _ in range(3):
        r.render_views(cams)
        glo, ghi, gval, ranges, ctl = r.read_back()
        cap = r.capacity()[0]
        assert ctl.status == 0 and ctl.ext_pad[0] > 0 and ctl.entries == cap < fctl.duplicates
        assert ctl.duplicates == fctl.duplicates and ctl.overflow == fctl.duplicates - cap
        if order is None:
            order = np.lexsort((hi, val, lo, view))[:cap]
            order = order[np.lexsort((val[order], lo[order], hi[order]))]
        np.testing.assert_array_equal(ghi, hi[order])
        np.testing.assert_array_equal(glo, lo[order])
        np.testing.assert_array_equal(gval, val[order])
        np.testing.assert_array_equal(ranges[:, 1] - ranges[:, 0], np.bincount(ghi, minlength=len(ranges)))
    r.close()
    gs.close()


@pytest.mark.parametrize("tile", [16, 8, 32])
@pytest.mark.parametrize("bounds", ["rect", "tight", "cutoff-only"])
@pytest.mark.parametrize("splat", ["full", "p24"])
@pytest.mark.parametrize("count,scale,away", [(20_000, 1.0, False), (3000, 30.0, False), (20_000, 1.0, True),
                                                (90_000, 1.0, True)])
def test_largest_tile_id_is_of_all_records(gpu, count, scale, away, bounds, tile, splat):
    """Kept or not, as in a sorted list; also where the last view sees nothing."""
    from gsr_b200 import scenes

    scene = tile_raster_scene(count, seed=count, needles=True)
    scene.scales[:] *= np.float32(scale)
    scene.pos_alpha[:, 1] += np.float32(0.5)  # off the middle: the last row is not always the image's
    gs = gpu.GpuScene(scene)
    cams = [scenes.viewer_camera((0.3 + k, 0.5, 6.0), (0.0, 0.0, 60.0) if away and k == 2 else (0.0, 0.0, 0.0), 640, 360, 60.0)
            for k in range(3)]
    kw = dict(adaptive_list=False, bounds=bounds, tile_size=tile, render_splat=splat)
    want = []
    for mode, mb in (("global", 2048), ("binning", 2048), ("binning", 1)):
        r = gpu.Renderer(gs, gpu.Settings(budget_mb=mb, list_mode=mode, **kw))
        for _ in range(2):
            r.render_views(cams)
        c = r.read_control()
        assert c.status == 0 and (mb == 1 or c.overflow == 0)
        if mb == 1 and count != 20_000:
            assert c.overflow > 0
        want.append((c.tile_max, c.duplicates, c.visible))
        if mode == "binning":
            assert c.key_bits == c.tile_max.bit_length() and c.ext_pad[0] > 0
        r.close()
    assert want[0] == want[1] == want[2]
    gs.close()
