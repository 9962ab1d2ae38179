"""The training step's weight image (kept by the Adam kernel) and its samples fetched a chunk ahead: runs
of k steps in one call and in several resumed calls (each of which makes the image anew from the
parameters) give the same parameters, moments and losses bit for bit, at the smallest batch (one
block), a ragged number of partial sums (no multiple of the 64 that Adam loads together) and scenes
smaller than a chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,degree,batch", [(1, 0, 256), (63, 1, 256), (5_000, 2, 256 * 65), (20_000, 3, 256 * 130)])
def test_one_call_equals_resumed_calls(gpu, tmp_path, count, degree, batch):
    from gsr_b200 import scenes

    gs = gpu.GpuScene(scenes.make_scene(count, seed=count, ball_radius=3.0, sh_degree=degree))

    def state(model):
        model.save(tmp_path / "m")
        ck = gpu.read_color_checkpoint(tmp_path / "m")
        return [ck[k] for k in ("params", "adam_m", "adam_v", "loss", "latents")]

    whole = gpu.ColorModel(gs, steps=7, batch=batch, seed=3)
    parts = gpu.ColorModel(gs, steps=1, batch=batch, seed=3)
    parts.resume(4)
    parts.resume(2)
    for a, b in zip(state(whole), state(parts)):
        assert a.tobytes() == b.tobytes()
    assert np.isfinite(state(whole)[0]).all() and whole.stats()["final_loss"] > 0.0
    whole.close()
    parts.close()
    gs.close()
