"""Frames of more than 2^32 tiles: the row-wise list is still the full one cut at its capacity in (depth,
gaussian, tile) order. The splats are placed so that the whole list is known: their depths order like their
indices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(count, x, scale, alpha):
    from gsr_b200 import scenes

    pos = np.zeros((count, 4), np.float32)
    pos[:, 0] = x
    pos[:, 2] = np.linspace(2.0, -2.0, count)  # the camera looks along -z from z = 6
    pos[:, 3] = alpha
    scales = np.zeros((count, 4), np.float32)
    scales[:, :3] = scale
    rotations = np.zeros((count, 4), np.float32)
    rotations[:, 0] = 1.0
    return scenes.Scene(pos, scales, rotations, np.zeros(count * 3, np.float32), 0)


def _frame(gpu, scene, width, height, bounds):
    from gsr_b200 import scenes

    gs = gpu.GpuScene(scene)
    r = gpu.Renderer(gs, gpu.Settings(adaptive_list=False, budget_mb=4, bounds=bounds))
    r.render(scenes.viewer_camera((0.0, 0.0, 6.0), (0.0, 0.0, 0.0), width, height, 60.0))
    _, hi, val, ranges, ctl = r.read_back()
    cap = r.capacity()[0]
    assert ctl.status == 0 and ctl.ext_pad[0] > 0, ctl.as_dict()
    assert ctl.duplicates == 0xFFFFFFFF and ctl.entries == cap and ctl.overflow == 0xFFFFFFFF - cap
    r.close()
    gs.close()
    return hi, val, ranges, cap


def _every_tile(gpu, count, width, height):
    """Splats that cover every tile: the list holds the first ones in every tile, the last of them in the
    tiles that are left."""
    hi, val, ranges, cap = _frame(gpu, _scene(count, 0.0, 60.0, 0.5), width, height, "rect")
    tiles = (width // 16) * (height // 16)
    of_tile = cap // tiles + (np.arange(tiles) < cap % tiles)
    end = np.cumsum(of_tile)
    np.testing.assert_array_equal(ranges, np.stack([end - of_tile, end], 1))
    np.testing.assert_array_equal(hi, np.repeat(np.arange(tiles), of_tile))
    np.testing.assert_array_equal(val, np.arange(cap) - np.repeat(end - of_tile, of_tile))


def test_prefix_past_32_bits(gpu):
    _every_tile(gpu, 4_300_000, 512, 512)  # 1,024 tiles each


def test_a_row_past_32_bits(gpu):
    _every_tile(gpu, 2 ** 23, 8192, 688)  # 512 tiles of each of the 43 rows: 2^32 a row


def test_more_spilled_runs_than_32_bits_count(gpu):
    """17.2 M needles over all 256 tile rows ask for 4.4 G spilled runs; the near half, of which the list's
    records are, is in the image's 16th tile column, the far half in its 17th."""
    count = 17_200_000
    x = np.where(np.arange(count) < count // 2, -0.009, 0.0135)
    scene = _scene(count, x, (0.001, 20.0, 0.001), 0.5)
    hi, val, ranges, cap = _frame(gpu, scene, 512, 4096, "tight")
    of_row = cap // 256 + (np.arange(256) < cap % 256)
    end = np.cumsum(of_row)
    want = np.zeros((256, 32, 2), np.uint32)
    want[:, 15] = np.stack([end - of_row, end], 1)
    np.testing.assert_array_equal(ranges, want.reshape(-1, 2))
    np.testing.assert_array_equal(hi, np.repeat(np.arange(256) * 32 + 15, of_row))
    np.testing.assert_array_equal(val, np.arange(cap) - np.repeat(end - of_row, of_row))
