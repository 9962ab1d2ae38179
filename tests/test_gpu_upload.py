"""The scene upload by several threads through page-locked slots (and the paths beside it: small scenes,
page-locked sources, a second upload at the same moment): the device buffers hold the host arrays bit
for bit, for totals that end inside a piece, on its boundary, and after the slots were given back."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(count, seed, degree=3):
    from gsr_b200 import scenes

    rng = np.random.default_rng(seed)
    K = (degree + 1) ** 2

    def words(*shape):
        return rng.integers(0x3F000000, 0x3FFFFFFF, shape, np.uint32).view(np.float32)

    return scenes.Scene(words(count, 4), words(count, 4), words(count, 4), words(count * K * 3), degree)


def _check(gpu, host, gs):
    for b, a in enumerate((host.pos_alpha, host.scales, host.rotations, host.sh)):
        assert np.array_equal(gs.buffer(b), a.reshape(-1).view(np.uint32)), b


@pytest.mark.parametrize("count", [1, 65_536, 279_620, 300_001, 2 ** 19])
def test_soa_buffers_hold_the_arrays(gpu, count):
    for again in range(2):  # the second time after the slots were given back
        host = _scene(count, count + again)
        gs = gpu.GpuScene(host)
        _check(gpu, host, gs)
        small = gpu.GpuScene(_scene(40_000, 7))  # with the slots in place
        small.close()
        gs.close()


def test_uploads_at_the_same_moment(gpu):
    hosts = [_scene(300_000 + 17 * k, k) for k in range(4)]
    got = [None] * len(hosts)

    def make(k):
        got[k] = gpu.GpuScene(hosts[k])

    threads = [threading.Thread(target=make, args=(k,)) for k in range(len(hosts))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for host, gs in zip(hosts, got):
        _check(gpu, host, gs)
        gs.close()


def test_page_locked_source(gpu):
    import torch

    host = _scene(300_000, 5)
    pinned = torch.from_numpy(host.sh).pin_memory()
    host.sh = pinned.numpy()
    gs = gpu.GpuScene(host)
    _check(gpu, host, gs)
    gs.close()
