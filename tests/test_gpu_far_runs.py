"""Very long, nearly horizontal splats that have left the image at some of their tile rows, so that the
row's run starts (empty) more than 1,048,576 pixels to its right: the rows' runs are packed in 16 bits an
end. The list against the oracle's, entry for entry, for every tile shape and both bounds that use the
ellipse, with runs in the hint, spilled runs, and more of those than the frame holds; between ordinary
splats, whose rows' entries must stay in their places."""
import numpy as np
import pytest

from helpers import tile_raster_scene


def _scene(needles, half_height):
    """`needles` splats of 12 half heights a radian / slope: their rows reach half_height pixels about."""
    scene = tile_raster_scene(3000, seed=23)
    n = np.arange(needles)
    slope = np.where(n % 2 == 0, 5e-6, 4e-6) * np.where(n % 3 == 0, -1.0, 1.0)
    at = slice(0, needles)
    scene.pos_alpha[at, 0] = (n % 7) * 0.1 - 0.3
    scene.pos_alpha[at, 1] = (n % 11) * 0.15 - 0.75
    scene.pos_alpha[at, 2] = (n % 13) * 0.01
    scene.pos_alpha[at, 3] = 0.9
    scene.scales[at, 0] = half_height / 3.4 / 52.0 / np.abs(slope)  # 52 pixels a unit at the scene's middle
    scene.scales[at, 1:3] = 0.001
    scene.rotations[at] = 0.0
    scene.rotations[at, 0] = 1.0
    scene.rotations[at, 3] = 0.5 * slope
    return scene


def _camera():
    from gsr_b200 import scenes

    return scenes.viewer_camera((0.0, 0.0, 6.0), (0.0, 0.0, 0.0), 640, 360, 60.0)


def _oracle(port, scene, bounds, tile):
    cam = _camera()
    ocam = port.camera_from_viewer(cam.view, cam.proj, cam.model, cam.width, cam.height)
    splats = port.preprocess(scene, ocam, scene.sh_degree, gpu_rules=True)
    counts = port.coverage_counts(splats, ocam, bounds, tile)
    return splats, counts, port.tile_list(splats, counts, ocam, bounds, tile)


def _far_rows(splats, tile):
    """Tile rows of the visible splats whose run starts past 1,048,576 pixels (64-bit estimate)."""
    high = 8 if tile == 32 else tile
    far = 0
    for s in splats[splats["cullReason"] == 0]:
        A, B, C, o = (float(v) for v in s["conicOpacity"])
        D, t = A * C - B * B, 2.0 * np.log(255.0 * float(o))
        if not (A > 0 and D > 0 and t > 0):
            continue
        half = np.sqrt(t * A / D)
        dy = np.arange(360 // high + 1)[:, None] * high + np.array([0.0, high - 1.0]) - float(s["center"][1])
        lo, hi = np.maximum(dy.min(1), -half), np.minimum(dy.max(1), half)
        at = np.stack([lo, hi], 1)[lo <= hi]
        if len(at):
            left = (-B * at - np.sqrt(np.maximum(0.0, A * t - D * at * at))) / A + float(s["center"][0])
            far += int((left.min(1) > 1.1 * 1048576.0).sum())
    return far


CASES = [(1, 25.0), (40, 25.0), (60, 170.0), (900, 170.0)]


@pytest.mark.parametrize("needles,half_height", CASES)
def test_the_scenes_reach_far_rows(port, needles, half_height):
    splats, _, _ = _oracle(port, _scene(needles, half_height), 1, 16)
    assert (splats["cullReason"][:needles] == 0).all()
    assert _far_rows(splats[:needles], 16) >= max(1, needles // 3)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [16, 8, 32])
@pytest.mark.parametrize("bounds", [1, 2])
@pytest.mark.parametrize("needles,half_height", CASES)
def test_list_is_the_oracles(gpu, port, needles, half_height, bounds, tile):
    scene = _scene(needles, half_height)
    _, counts, want = _oracle(port, scene, bounds, tile)
    gs = gpu.GpuScene(scene)
    for mode in ("binning", "global"):
        r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, bounds=("rect", "tight", "cutoff-only")[bounds], tile_size=tile,
                                          list_mode=mode, budget_mb=512))
        r.render(_camera())
        lo, hi, val, ranges, ctl = r.read_back()
        assert ctl.status == 0 and ctl.coverage_mismatch == 0, ctl.as_dict()
        np.testing.assert_array_equal(r.read_back_splats(scene.count)[1], counts)
        np.testing.assert_array_equal(hi, want["keys_hi"])
        np.testing.assert_array_equal(lo, want["keys_lo"])
        np.testing.assert_array_equal(val, want["values"])
        np.testing.assert_array_equal(ranges, want["ranges"])
        r.close()
    gs.close()
