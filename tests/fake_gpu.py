"""The library's host side (renderer.cpp) over tests/fake_gpu.cpp: no device, calls that can be made to fail."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

import gsr_b200

REPO = Path(__file__).resolve().parents[1]
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))


@pytest.fixture(scope="session")
def fake_library(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake_gpu") / "libgsr_fake.so"
    csrc = REPO / "gaussian-splat-renderer_b200" / "csrc"
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-pthread", f"-I{REPO / 'include'}", f"-I{csrc}",
                    f"-I{CUDA / 'include'}", "-o", out, csrc / "renderer.cpp", csrc / "color_checkpoint.cpp",
                    REPO / "tests" / "fake_gpu.cpp", "-Wl,-z,defs,-Bsymbolic"], check=True)
    return out


@pytest.fixture
def fake(fake_library, monkeypatch):
    """gsr_b200 over the fake library; what a test makes is closed by the test."""
    monkeypatch.setattr(gsr_b200, "_lib", None)
    monkeypatch.setattr(gsr_b200, "LIB_PATH", fake_library)
    lib = gsr_b200.load(build_if_missing=False)
    lib.fake_fail.argtypes = [C.c_char_p, C.c_int]
    lib.fake_page_locked.argtypes = [C.c_void_p, C.c_size_t]
    lib.fake_live_bytes.restype = C.c_size_t
    yield lib
    for name in (b"cudaMalloc", b"cudaHostAlloc", b"cudaMemcpy", b"cudaMemcpyAsync", b"cudaStreamCreateWithFlags",
                 b"cudaEventCreateWithFlags"):
        lib.fake_fail(name, 0)
