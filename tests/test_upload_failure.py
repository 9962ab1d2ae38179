"""The threaded scene upload when one of its threads, or all of them, cannot set up a stream or an event,
or the slots cannot be page-locked: the scene holds the arrays all the same (a failed transfer is reported).
An upload with any page-locked array is a plain copy, in the order of the work before it."""
import numpy as np
import pytest

import gsr_b200
from fake_gpu import fake, fake_library  # noqa: F401  (fixtures)


@pytest.fixture(scope="module")
def host():
    from gsr_b200 import scenes

    rng = np.random.default_rng(1)
    n = 300_001  # 72 MB: the slots are made for it

    def words(*shape):
        return rng.integers(0x3F000000, 0x3FFFFFFF, shape, np.uint32).view(np.float32)

    return scenes.Scene(words(n, 4), words(n, 4), words(n, 4), words(n * 48), 3)


def _check(host):
    gs = gsr_b200.GpuScene(host)
    for b, a in enumerate((host.pos_alpha, host.scales, host.rotations, host.sh)):
        assert np.array_equal(gs.buffer(b), a.reshape(-1).view(np.uint32)), b
    gs.close()


@pytest.mark.parametrize("call,nth", [("cudaStreamCreateWithFlags", k) for k in (1, 2, 4, -1, -2)]
                         + [("cudaEventCreateWithFlags", k) for k in (1, 2, 3, 8, -1, -3)] + [("cudaHostAlloc", 1)])
def test_failed_set_up(fake, host, call, nth):  # noqa: F811
    fake.fake_fail(call.encode(), nth)
    _check(host)
    fake.fake_fail(call.encode(), 0)
    _check(host)


@pytest.mark.parametrize("nth", [1, 5, -1])
def test_failed_transfer(fake, host, nth):  # noqa: F811
    fake.fake_fail(b"cudaMemcpyAsync", nth)
    with pytest.raises(gsr_b200.GsrError):
        gsr_b200.GpuScene(host)
    fake.fake_fail(b"cudaMemcpyAsync", 0)
    _check(host)


@pytest.mark.parametrize("array", ["pos_alpha", "scales", "rotations", "sh"])
def test_a_page_locked_array(fake, host, array):  # noqa: F811
    a = getattr(host, array)
    fake.fake_page_locked(a.ctypes.data, a.nbytes)
    before = fake.fake_calls(b"cudaMemcpyAsync"), fake.fake_calls(b"cudaHostAlloc")
    _check(host)
    assert before == (fake.fake_calls(b"cudaMemcpyAsync"), fake.fake_calls(b"cudaHostAlloc"))
    fake.fake_page_locked(a.ctypes.data, 0)
