"""The host layer's decisions (capi.cpp) against a CUDA runtime that only keeps books (fake_cuda.cpp): what a call
does when a capture, an allocation or a launch fails, which memory is held when, and what the autotuners pick
when the costs are known."""
import ctypes
import os
import subprocess

import pytest

from mrlbm_2d_b200 import api
from mrlbm_2d_b200.config import cylinder_case

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mrlbm_2d_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"
STEP, PAIR, BATCH = 0, 1, 2

pytestmark = pytest.mark.skipif(not os.path.isdir(CUDA_INC), reason="CUDA headers not installed")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    srcs = [os.path.join(CSRC, f) for f in ("capi.cpp", "geometry.cpp", "statistics.cpp")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", CUDA_INC,
                    *srcs, os.path.join(ROOT, "tests", "fake_cuda.cpp"), "-o", out], check=True)
    L = api.load_library(out)
    for f in ("fake_used", "fake_peak", "fake_done", "fake_captures", "fake_dangling"):
        getattr(L, f).restype = ctypes.c_int64
    return L


@pytest.fixture
def fake(library, monkeypatch):
    monkeypatch.setattr(api, "_lib", library)
    monkeypatch.delenv("MRLBM_PAIRS", raising=False)
    library.fake_reset()
    yield library
    assert library.fake_dangling() == 0


def small():
    return cylinder_case(120, 48, 12, 30.0, 24.5, 100.0, 0.05)


def large():
    """Above the size from which FP64 steps are taken in pairs."""
    return cylinder_case(1400, 520, 40, 300.0, 260.5, 100.0, 0.05)


def level_bytes(s):
    return s.info.state_bytes


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("call", ["cudaMalloc", "cudaStreamBeginCapture", "launch", "cudaStreamEndCapture", "cudaGraphInstantiate",
                                  "cudaMemcpyAsync", "cudaGraphLaunch"])
def test_a_replay_that_cannot_be_made_is_launched_step_by_step(fake, prec, call):
    s = api.Simulation(small(), precision=prec)
    fake.fake_fail(call.encode(), 1)                         # the first call of its kind is the replay's
    s.step(2600)
    assert s.iter == 2601 and fake.fake_done(STEP) == 2600
    captures = fake.fake_captures()
    s.step(2600)                                             # not tried again for every run
    assert fake.fake_captures() == captures and fake.fake_done(STEP) == 5200
    s.close()
