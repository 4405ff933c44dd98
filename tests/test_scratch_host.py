"""The scratch of the library's host calls (kma_scratch.cu) over a made-up
CUDA runtime (tests/scratch_fake.cpp): contexts, resets, limits.  No GPU."""
import os
import shutil
import subprocess

import pytest

from kma_b200 import build as kbuild

HERE = os.path.dirname(os.path.abspath(__file__))
SCENARIOS = ["contexts", "reset", "two_devices", "capture", "no_host_memory", "bounded"]


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cxx = os.environ.get("CXX", "g++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(kbuild.nvcc()))), "include")
    if shutil.which(cxx) is None or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    binary = str(tmp_path_factory.mktemp("scratch") / "fake")
    subprocess.run([cxx, "-O1", "-std=c++17", "-w", "-I", cuda, "-I", kbuild.CSRC, "-I", kbuild.INCLUDE, "-x", "c++",
                    os.path.join(kbuild.CSRC, "kma_scratch.cu"), os.path.join(HERE, "scratch_fake.cpp"),
                    "-o", binary, "-pthread"], check=True)
    return binary


@pytest.mark.parametrize("scenario", SCENARIOS)
def test_scratch(fake, scenario):
    r = subprocess.run([fake, scenario], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
