"""The wait for a block's SH copy before its rows are shared out through the same shared memory: when it
expires (forced by the test hook, for every block), the splats get no tiles, the records are those of the
undisturbed frame, the frame reports the timeout, and the next frame is whole again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["binning", "global"])
@pytest.mark.parametrize("count", [200, 30_001])
def test_expired_wait_leaves_no_tiles(gpu, mode, count):
    from gsr_b200 import scenes

    scene = scenes.make_scene(count, seed=4, ball_radius=2.0)  # degree 3: the staged colours
    scene.scales[::50, 1] *= 40.0  # splats of many rows
    cam = scenes.viewer_camera((0.3, 0.5, 6.0), (0.0, 0.0, 0.0), 640, 360, 60.0)
    gs = gpu.GpuScene(scene)
    r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, list_mode=mode))
    r.render(cam)
    good, (splats, counts) = r.read_back(), r.read_back_splats(count)
    assert good[4].status == 0 and good[4].entries > 0
    r.force_timeout(64)
    r.render(cam)
    c = r.read_control()
    assert c.status & gpu.CONTROL_TIMEOUT and c.entries == 0 and c.duplicates == 0, c.as_dict()
    forced, none = r.read_back_splats(count)
    visible = splats["cullReason"] == 0
    assert not none.any() and forced[visible].tobytes() == splats[visible].tobytes()
    r.render(cam)
    again = r.read_back()
    assert again[4].status == 0
    for a, b in zip(good[:4], again[:4]):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(r.read_back_splats(count)[1], counts)
    r.close()
    gs.close()
