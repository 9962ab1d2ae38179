"""The rasterizer's two pixels a thread and its walk over pairs of listed records: against the stats
build (one pixel a thread, one record at a time), bit for bit, and against the oracle's image. List
lengths around the batch (128 entries), the 32-record group and the pair; image widths that end
inside a tile, a strip and a pixel pair; records that reach the 0.99 cap (opacity up to 1, wide
footprints over the whole image) and needles."""
import numpy as np
import pytest

from helpers import oracle_frame, psnr, tile_raster_scene

pytestmark = pytest.mark.gpu


def _scene(count, opaque):
    s = tile_raster_scene(max(count, 1), seed=count, needles=True)
    s.pos_alpha[:, :3] *= np.float32(0.15)  # in front of the camera, on few tiles
    if opaque:
        s.pos_alpha[:, 3] = np.float32(1.0) - np.float32(0.02) * (np.arange(count) % 3)
    return s


@pytest.mark.parametrize("count,size", [(1, (17, 9)), (2, (16, 16)), (31, (31, 33)), (33, (8, 47)), (64, (49, 15)),
                                        (127, (15, 16)), (129, (33, 17)), (257, (64, 31)), (3000, (97, 65))])
@pytest.mark.parametrize("tile", [16, 32])
@pytest.mark.parametrize("opaque", [False, True])
def test_pairs_equal_the_one_pixel_walk(gpu, port, count, size, tile, opaque):
    from gsr_b200 import scenes

    scene = _scene(count, opaque)
    cam = scenes.viewer_camera((0.3, 0.5, 6.0), (0.0, 0.0, 0.0), size[0], size[1], 30.0)
    gs = gpu.GpuScene(scene)
    images = []
    for stats in (False, True):
        r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, rgb8=True, tile_size=tile, tile_stats=stats))
        r.render(cam)
        assert r.read_control().status == 0
        images.append(r.read_back_image(rgb8=True))
        r.close()
    assert images[0][0].tobytes() == images[1][0].tobytes()
    assert images[0][1].tobytes() == images[1][1].tobytes()
    ocam, _, _, _ = oracle_frame(port, scene, cam)
    ref, _ = port.render(scene, ocam, bounds=1)
    assert psnr(images[0][0][..., :3], ref) > 60.0
    gs.close()
