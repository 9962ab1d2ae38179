"""An allocation that fails while a renderer's layout is set up, at each allocation in turn: the call
reports it, and so does every later call until the layout is complete; no launch is ever handed a missing
buffer, and a call after the failure that finds memory again renders."""
import numpy as np
import pytest

import gsr_b200
from fake_gpu import fake, fake_library  # noqa: F401  (fixtures)
from helpers import tile_raster_scene


def _cams(sizes):
    from gsr_b200 import scenes

    return [scenes.viewer_camera((0.3, 0.5, 6.0), (0.0, 0.0, 0.0), w, h, 60.0) for w, h in sizes]


FIRST = [(640, 360)]  # row by row, 2 passes of a sorted list's tile ids
LAYOUTS = {"sorted, as many passes": [(16, 4097)], "sorted, more views": [(16, 4097), (640, 360)],
           "row by row, more views": [(640, 360), (320, 180)], "more passes": [(4096, 4096)], "sorted, more passes": [(8208, 4112)]}


@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("mode", ["binning", "global"])
def test_every_allocation_in_turn(fake, layout, mode):  # noqa: F811
    gs = gsr_b200.GpuScene(tile_raster_scene(2000, seed=1))
    first, second = _cams(FIRST), _cams(LAYOUTS[layout])
    failures = 0
    for nth in range(1, 100):
        r = gsr_b200.Renderer(gs, gsr_b200.Settings(adaptive_list=False, list_mode=mode, budget_mb=8))
        r.render_views(first)
        fake.fake_fail(b"cudaMalloc", nth)
        try:
            r.render_views(second)
        except gsr_b200.GsrError as e:
            assert e.status == 4
            failures += 1
        else:
            break
        finally:
            fake.fake_fail(b"cudaMalloc", 0)
        fake.fake_fail(b"cudaMalloc", 1)  # still no memory for the next one
        with pytest.raises(gsr_b200.GsrError):
            for _ in range(2):
                r.render_views(second)
        fake.fake_fail(b"cudaMalloc", 0)
        for cams in (second, first, second):
            r.render_views(cams)
            r.read_back()
        assert fake.fake_null_launches() == 0
        r.close()
    else:
        pytest.fail("every allocation failed")
    assert failures >= 3
    r.close()
    gs.close()


def test_the_old_layout_after_a_failure(fake):  # noqa: F811
    """The layout that was complete before the failure is set up again, not used with what is left of it."""
    gs = gsr_b200.GpuScene(tile_raster_scene(2000, seed=1))
    sorted_form, more = _cams([(16, 4097)]), _cams([(640, 360), (320, 180)])
    for nth in range(1, 40):
        r = gsr_b200.Renderer(gs, gsr_b200.Settings(adaptive_list=False, budget_mb=8))
        r.render_views(sorted_form)
        fake.fake_fail(b"cudaMalloc", nth)
        try:
            r.render_views(more)
            break
        except gsr_b200.GsrError:
            pass
        finally:
            fake.fake_fail(b"cudaMalloc", 0)
        r.render_views(sorted_form)
        assert fake.fake_null_launches() == 0
        assert np.array_equal([(v.width, v.height) for v in r.view_layouts()], [(16, 4097)])
        r.close()
    r.close()
    gs.close()


@pytest.mark.parametrize("views", [1, 3])
def test_a_sorted_layout_holds_no_row_wise_scratch(fake, views):  # noqa: F811
    """Device memory of a sorted layout, against the global mode's: the depth sort's words and no more a
    gaussian; after a row-wise layout in between the same again."""
    count = 200_000
    gs = gsr_b200.GpuScene(tile_raster_scene(count, seed=1))
    start = fake.fake_live_bytes()
    sorted_form, rows = _cams([(16, 4097)] * views), _cams([(640, 360)] * views)
    held = {}
    for mode in ("global", "binning"):
        r = gsr_b200.Renderer(gs, gsr_b200.Settings(adaptive_list=False, list_mode=mode, budget_mb=8))
        r.render_views(sorted_form)
        held[mode] = fake.fake_live_bytes() - start
        if mode == "binning":
            r.render_views(rows)
            assert fake.fake_live_bytes() - start > held[mode]
            r.render_views(sorted_form)
            assert fake.fake_live_bytes() - start == held[mode]
        r.close()
        assert fake.fake_live_bytes() == start
    depth_sort = views * (count * 16 + 4 * -(-count // 4096) * 256 * 8 + 2 * 4 * 4 * 256)
    assert held["binning"] - held["global"] < depth_sort + 64 * 1024
    gs.close()
