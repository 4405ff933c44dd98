"""Device calls with the options a user's own kernels give them, which the
library's entry points do not reach (tests/device_calls.cu, built here)."""
import ctypes
import os
import re
import shutil
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


def test_per_thread_dequeues_fit_a_block_of_1024_threads(tmp_path):
    """They are header code in the user's kernel: with more than 64 registers
    a thread, or arrays in local memory, a kernel of one such call would not
    launch with 1024 threads, or would pay for what its lanes never use."""
    if shutil.which(kbuild.nvcc()) is None:
        pytest.skip("no nvcc")
    r = subprocess.run([kbuild.nvcc(), *kbuild.ARCH, "-O3", "-std=c++17", "-Xptxas", "-v", "-I", kbuild.INCLUDE, "-c",
                        "-o", str(tmp_path / "o.o"), os.path.join(HERE, "device_calls.cu")],
                       check=True, capture_output=True, text=True)
    found = re.findall(r"Compiling entry function '\w*(k_user_\w+?queue)\w*'.*?(\d+) bytes stack frame.*?Used (\d+) registers",
                       r.stderr, re.S)
    assert {f[0] for f in found} == {"k_user_clqueue", "k_user_iqueue"}
    for name, stack, regs in found:
        assert int(stack) == 0 and int(regs) <= 64, (name, stack, regs)


def _lanes(calls, nq, n, stuck, step):
    import torch
    q = torch.zeros(2 * nq, dtype=torch.int64, device="cuda")
    items = torch.zeros(2 * nq * n, dtype=torch.int64, device="cuda")
    out = torch.full((32,), -7, dtype=torch.int32, device="cuda")
    err = torch.zeros(32, dtype=torch.int32, device="cuda")
    rc = calls.t_lanes_dequeue(ctypes.c_void_p(q.data_ptr()), ctypes.c_void_p(items.data_ptr()), nq, n, stuck, step,
                               ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(err.data_ptr()))
    assert rc == 0
    return out.cpu().numpy(), err.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("step", [0, 5])
@pytest.mark.parametrize("nq,n", [(1, 1), (1, 20), (1, 32), (1, 40), (2, 9), (2, 16), (3, 20)])
def test_lanes_of_a_warp_dequeue_each_its_own(calls, nq, n, step):
    """On one queue or several, with one limit or several: the first items
    come out, each to one lane, and nobody's wait is reported as expired."""
    out, err = _lanes(calls, nq, n, 0, step)
    assert not err.any()
    for k in range(nq):
        mine = out[k::nq]
        assert sorted(mine[mine >= 0]) == list(range(min(n, len(mine))))
        assert (mine >= -1).all()


@pytest.mark.gpu
@pytest.mark.parametrize("step", [0, 5])
@pytest.mark.parametrize("nq", [1, 2])
def test_every_lane_learns_of_its_expired_wait(calls, nq, step):
    """A head that is never given back: each lane gets NULL, and the timeout
    in the error word that it passed."""
    from kma_b200 import KMA_FLAG_TIMEOUT
    out, err = _lanes(calls, nq, 3, 1, step)
    assert (out == -1).all() and ((err & KMA_FLAG_TIMEOUT) != 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("shards,at,other", [(2, 0, 1), (9, 0, 8), (9, 3, 2), (66, 0, 1), (66, 0, 7), (66, 0, 8), (66, 0, 9),
                                             (66, 0, 63), (66, 0, 64), (66, 0, 65), (66, 40, 9), (66, 65, 0)])
def test_an_exhausted_heap_serves_from_the_next_64_shards(calls, shards, at, other):
    """The free list is empty and shard `other` has a superblock with slots
    left: per-thread calls of shard `at` get all of them, if it is near enough."""
    import torch
    from kma_b200 import Heap, slots_by_size
    n = 32
    with Heap(shards * 32 + 1, 12, shards=shards) as h:
        got = torch.zeros(1, dtype=torch.int32, device="cuda")

        def malloc_at(shard, size, count):
            rc = calls.t_malloc_at(ctypes.c_void_p(h.device_ptr), shard // 8, shard % 8, size, count,
                                   ctypes.c_void_p(got.data_ptr()))
            assert rc == 0
            return int(got[0])

        assert malloc_at(other, n, 1) == 1
        full = malloc_at(at, 4000, 1 << 20)  # one block to a superblock: the free list runs empty
        assert 0 < full < 1 << 20
        near = 1 <= (other - at) % shards <= 64
        assert malloc_at(at, n, 1 << 20) == (slots_by_size(12, n) - 1 if near else 0)
        assert malloc_at(at, n, 1) == 0
        assert h.error_flags() == 0
