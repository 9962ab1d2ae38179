"""Frames of few tiles have one pixel a thread, others two: the same images, bit for bit, on either side of
the line (512 tiles, reached by many views of a small image), against the stats build (one pixel a thread,
one record at a time). Image widths that end inside a tile, a strip and a pixel pair; list lengths around
the batches of both forms (256 and 128 entries); both schedules and gathers, every record format."""
import numpy as np
import pytest

from helpers import tile_raster_scene

pytestmark = pytest.mark.gpu


def _scene(count, opaque):
    s = tile_raster_scene(count, seed=count + 1, needles=True)
    s.pos_alpha[:, :3] *= np.float32(0.15)  # in front of the camera, on few tiles
    if opaque:
        s.pos_alpha[:, 3] = np.float32(1.0) - np.float32(0.02) * (np.arange(count) % 3)
    return s


def _images(gpu, gs, cams, views, **kw):
    r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, rgb8=True, budget_mb=512, **kw))
    r.render_views(cams[:views])
    c = r.read_control()
    assert c.status == 0 and c.overflow == 0 and c.entries > 0
    out = [r.read_view_image(v, rgb8=True) for v in (0, views // 2, views - 1)]
    r.close()
    return [b"".join(x.tobytes() for x in image) for image in out]


@pytest.mark.parametrize("count,size", [(1, (17, 9)), (2, (16, 16)), (33, (31, 33)), (64, (8, 47)), (129, (49, 15)),
                                        (255, (33, 17)), (513, (64, 31)), (3000, (97, 65))])
@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("opaque", [False, True])
def test_either_side_of_the_line(gpu, count, size, tile, opaque):
    from gsr_b200 import scenes

    tiles = -(-size[0] // tile) * -(-size[1] // (8 if tile == 32 else 16))
    few = 512 // tiles
    cams = [scenes.viewer_camera((0.3 + 0.01 * (k % 7), 0.5, 6.0), (0.0, 0.0, 0.0), *size, 30.0) for k in range(few + 1)]
    gs = gpu.GpuScene(_scene(count, opaque))
    for views in (1, few, few + 1):
        want = _images(gpu, gs, cams, views, tile_size=tile, tile_stats=True)
        for schedule in ("per-tile", "persistent"):
            assert _images(gpu, gs, cams, views, tile_size=tile, raster_schedule=schedule) == want, (views, schedule)
    gs.close()


@pytest.mark.parametrize("kw", [dict(raster_gather="tma"), dict(render_splat="p32"), dict(render_splat="p24"),
                                dict(bounds="rect"), dict(target="rgba16f"), dict(list_mode="global")], ids=str)
@pytest.mark.parametrize("tile", [16, 32])
def test_forms(gpu, kw, tile):
    """One view alone (few tiles) and the same view among enough others."""
    from gsr_b200 import scenes

    cam = scenes.viewer_camera((0.3, 0.5, 6.0), (0.0, 0.0, 0.0), 97, 65, 30.0)
    gs = gpu.GpuScene(_scene(3000, False))
    assert _images(gpu, gs, [cam], 1, tile_size=tile, **kw)[0] == _images(gpu, gs, [cam] * 20, 20, tile_size=tile, **kw)[1]
    gs.close()


def test_the_line_of_many_gaussians(gpu):
    """1,024 and 1,025 tiles of 65,536 gaussians."""
    from gsr_b200 import scenes

    gs = gpu.GpuScene(_scene(65_536, False))
    cams = [scenes.viewer_camera((0.3, 0.5, 6.0), (0.0, 0.0, 0.0), 512, 512, 30.0),
            scenes.viewer_camera((0.3, 0.5, 6.0), (0.0, 0.0, 0.0), 9, 16, 30.0)]
    for views in (1, 2):
        assert _images(gpu, gs, cams, views) == _images(gpu, gs, cams, views, tile_stats=True)
    gs.close()
