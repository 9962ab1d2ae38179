"""The depth sort of short runs (one cluster a view, the words in its shared memory): the binning list
against the global mode's sorted list, entry for entry, at the edges of a warp's, a block's and the
cluster's share of words (1,024, 2,048 and 4,096 words a block), one past its 32,768 records and 12 views,
with equal depths (their order is the records') and views that see nothing."""
import numpy as np
import pytest

from helpers import tile_raster_scene

pytestmark = pytest.mark.gpu


def _compare(gpu, gs, cams, **kw):
    out = []
    for mode in ("binning", "global"):
        r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, list_mode=mode, budget_mb=512, **kw))
        for _ in range(2):  # the second frame reuses every buffer
            r.render_views(cams)
        ctl = r.read_control()
        assert ctl.status == 0 and ctl.overflow == 0, ctl.as_dict()
        out.append((r.read_back(), r.read_back_image(), ctl.visible))
        r.close()
    for a, b in zip(out[0][0][:4], out[1][0][:4]):
        np.testing.assert_array_equal(a, b)
    assert out[0][1].tobytes() == out[1][1].tobytes() and out[0][2] == out[1][2]
    return out[0][2]


def _cams(views, away=()):
    from gsr_b200 import scenes

    return [scenes.viewer_camera((6.0 * np.sin(k), 0.5, 6.0 * np.cos(k)),
                                 (12.0 * np.sin(k), 1.0, 12.0 * np.cos(k)) if k in away else (0.0, 0.0, 0.0),
                                 200 + 16 * k, 120, 60.0) for k in range(views)]


@pytest.mark.parametrize("count", [1, 31, 1023, 1024, 1025, 8191, 8192, 8193, 16384, 16385, 32767, 32768, 32769])
def test_run_lengths(gpu, count):
    gs = gpu.GpuScene(tile_raster_scene(count, seed=count))
    _compare(gpu, gs, _cams(1))


@pytest.mark.parametrize("digit_bits", [7, 8, 9])
@pytest.mark.parametrize("views", [2, 12, 13])
def test_runs(gpu, views, digit_bits):
    gs = gpu.GpuScene(tile_raster_scene(2500, seed=7))
    _compare(gpu, gs, _cams(views, away=(1,)), sort_digit_bits=digit_bits)


@pytest.mark.parametrize("depths", [1, 3])
def test_equal_depths(gpu, depths):
    scene = tile_raster_scene(9000, seed=11)
    scene.pos_alpha[:, 2] = np.arange(9000) % depths
    gs = gpu.GpuScene(scene)
    from gsr_b200 import scenes

    assert _compare(gpu, gs, [scenes.viewer_camera((0.0, 0.0, 6.0), (0.0, 0.0, 0.0), 200, 120, 60.0)]) > 0


def test_nothing_visible(gpu):
    scene = tile_raster_scene(5000, seed=3)
    scene.pos_alpha[:, 2] = -np.abs(scene.pos_alpha[:, 2])  # behind the camera, which looks along +z from z = 6
    gs = gpu.GpuScene(scene)
    assert _compare(gpu, gs, _cams(1, away=(0,))) == 0
