"""The window's slots in shared memory (K <= 16): every capacity (4, 8, 16) full and with unused slots,
fewer splats than K, in all three tile shapes, against the CPU reference with the same window (its own
bar, 60 dB) and the same image from every tile shape."""
import pytest

from helpers import oracle_frame, psnr, tile_raster_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 3, 5, 7, 8, 9, 15, 16])
@pytest.mark.parametrize("count", [3, 20_000])
def test_slots_match_the_cpu_window(gpu, port, K, count):
    from gsr_b200 import scenes

    scene = tile_raster_scene(count, seed=31, needles=True)
    cam = scenes.viewer_camera((0.3, 0.5, 6.0), (0.0, 0.0, 0.0), 131, 75)
    gs = gpu.GpuScene(scene)
    images = []
    for tile in (16, 8, 32):
        r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, sort_window=K, tile_size=tile))
        r.render(cam)
        assert r.read_control().status == 0
        images.append(r.read_back_image())
        r.close()
    assert images[0].tobytes() == images[1].tobytes() == images[2].tobytes()
    ocam, _, _, _ = oracle_frame(port, scene, cam)
    ref, _ = port.render(scene, ocam, bounds=1, sort_window=K)
    assert psnr(images[0][..., :3], ref) > 60.0
    gs.close()
