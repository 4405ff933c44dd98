"""Device calls with the options a user's own kernels give them, which the
library's entry points do not reach (tests/device_calls.cu, built here)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
from opstream import make_stream

from kma_b200 import build as kbuild

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def calls(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("calls") / "calls.so")
    subprocess.run([kbuild.nvcc(), *kbuild.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", kbuild.INCLUDE, "-o", so, os.path.join(HERE, "device_calls.cu")], check=True)
    return ctypes.CDLL(so)


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_one_lane_with_hints_replays_as_the_reference(calls, seed):
    """A single calling lane takes the reference's blocks, hints or not: a
    superblock that left its class slot is not reserved from."""
    import torch
    from kma_b200 import Heap
    from oracle import oracle
    ops = make_stream(seed, 3000, 12)
    with oracle.Port(64, 12) as p:
        want = p.replay(ops)
    with Heap(64, 12) as h:
        d = torch.from_numpy(ops).cuda()
        out = torch.full((len(ops),), -7, dtype=torch.int64, device="cuda")
        rc = calls.t_replay_hint(ctypes.c_void_p(h.device_ptr), ctypes.c_void_p(d.data_ptr()),
                                 ctypes.c_longlong(len(ops)), ctypes.c_void_p(out.data_ptr()))
        assert rc == 0
        np.testing.assert_array_equal(out.cpu().numpy(), want)
        assert h.error_flags() == 0
