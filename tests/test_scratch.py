"""The scratch that the library's host calls share (kma_scratch.h): calls of
several threads at once do not meet in one buffer, what stays is bounded, and
destroying a heap gives it back."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _queue(structs, kind, threads, per, bad):
    st = structs.c3_queue(kind, threads, per, 1, seed=threads)
    n = threads * per
    if not (st["err"] == 0 and st["walk_ok"] == 1 and st["out_count"] == n and st["out_sum"] == n * (n - 1) // 2):
        bad.append((kind, threads, per, st))


def _tree(structs, n, bad):
    keys = np.random.default_rng(n).permutation(n).astype(np.uint32)
    res, st = structs.c3_tree(np.zeros(n, np.uint8), keys, threads=max(1, n // 8))
    if not ((res == 1).all() and st["live_keys"] == n and st["keys_sum"] == n * (n - 1) // 2 and st["sorted"] == 1):
        bad.append((n, st))


def test_concurrent_calls_have_buffers_of_their_own():
    from kma_b200 import structs
    bad = []
    todo = [(_queue, structs, structs.C3_CLQUEUE | structs.C3_BLOCK, 2000 + 37 * i, 5, bad) for i in range(4)]
    todo += [(_queue, structs, structs.C3_IQUEUE | structs.C3_WARP, 3000 + 41 * i, 4, bad) for i in range(4)]
    todo += [(_tree, structs, 5000 + 999 * i, bad) for i in range(4)]
    for _ in range(3):
        ts = [threading.Thread(target=t[0], args=t[1:]) for t in todo]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    assert bad == []


@pytest.mark.parametrize("threads,per,kept", [(1 << 17, 64, True), (1 << 20, 80, False)])
def test_kept_scratch_is_bounded_and_given_back(threads, per, kept):
    from kma_b200 import Heap, structs
    with Heap(64, 12):
        pass
    before = _free()
    structs.c3_queue(structs.C3_IQUEUE, threads, per, 4096)  # 16 bytes a payload
    after = _free()
    size = threads * per * 16
    if kept:
        assert before - after >= size
    else:
        assert before - after < 1 << 28  # larger than what is ever kept
    assert before - after <= (1 << 30) + (64 << 20)
    with Heap(64, 12):
        pass
    assert before - _free() < 64 << 20


def test_a_program_gets_the_scratch_back():
    """For an allocation that is not the library's: no heap is destroyed."""
    import kma_b200
    from kma_b200 import structs
    kma_b200.trim_scratch()
    before = _free()
    structs.c3_queue(structs.C3_CLQUEUE, 1 << 17, 64, 4096)  # 16 bytes a payload
    assert before - _free() >= (1 << 23) * 16
    kma_b200.trim_scratch()
    assert before - _free() < 64 << 20
