"""The graph-build workload (include/kma_graph.h) after test/tb_clTree.cl:
one thread gives the reference's graph block for block (node offsets,
keys, every node's links in queue order); many threads give the same
multiset of edges, a search tree, and an empty heap after teardown."""
import os
from collections import defaultdict

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLD = np.load(os.path.join(ROOT, "tests", "golden", "structs.npz"))
SEEDS = sorted({k.split("_")[1] for k in GOLD.files if k.startswith("graph_")})


def edge_mix(a: np.ndarray, b: np.ndarray) -> np.ndarray:
    """mix(source, sink) as the library computes it (SplitMix64 finaliser of
    source << 32 | sink)."""
    with np.errstate(over="ignore"):
        z = (a.astype(np.uint64) << np.uint64(32) | b.astype(np.uint64)) + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


@pytest.mark.parametrize("seed", SEEDS)
def test_graph_fixture_is_edges_in_order(seed):
    """The reference's serial build: each source's links are its edges' sinks
    in edge order, and the nodes are the distinct endpoints."""
    e = GOLD[f"graph_{seed}_edges"]
    keys, sinks, start = GOLD[f"graph_{seed}_keys"], GOLD[f"graph_{seed}_sinks"], GOLD[f"graph_{seed}_start"]
    d = defaultdict(list)
    for a, b in e:
        d[int(a)].append(int(b))
    np.testing.assert_array_equal(keys, np.unique(e))
    for i, k in enumerate(keys):
        assert sinks[start[i]:start[i + 1]].tolist() == d.get(int(k), [])


def test_edge_mix_matches_library():
    from kma_b200 import graph
    a = np.array([0, 1, 0xFFFFFFFF, 12345], np.uint32)
    b = np.array([0, 2, 7, 0xFFFFFFFF], np.uint32)
    assert [graph.edge_mix(int(x), int(y)) for x, y in zip(a, b)] == edge_mix(a, b).tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("seed", SEEDS)
def test_gpu_graph_serial_equals_reference(seed):
    from kma_b200 import Heap, graph
    sblocks = int(GOLD[f"graph_{seed}_cfg"][0])
    e = GOLD[f"graph_{seed}_edges"].astype(np.uint32)
    with Heap(sblocks, 12) as h:
        st, (keys, offs, sinks, start) = graph.build(h, e, threads=1, free_after=True, export=True)
        np.testing.assert_array_equal(keys, GOLD[f"graph_{seed}_keys"])
        np.testing.assert_array_equal(offs, GOLD[f"graph_{seed}_offs"])
        np.testing.assert_array_equal(sinks, GOLD[f"graph_{seed}_sinks"])
        np.testing.assert_array_equal(start, GOLD[f"graph_{seed}_start"])
        assert st["lost_adds"] == 0 and st["nulls"] == 0 and st["err"] == 0 and st["sorted"] == 1
        from kma_b200 import inspect as ins
        assert ins.check_canonical_empty(h.snapshot(), h.bitmaps()) == []


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [4096, 65536])
def test_gpu_graph_concurrent_conserves_edges(threads):
    from kma_b200 import Heap, graph
    from kma_b200 import inspect as ins
    e = graph.synth_edges(77, 200_000, 20_000)
    with Heap(4096, 14) as h:
        st, _ = graph.build(h, e, threads=threads, free_after=True)
        m = edge_mix(e[:, 0], e[:, 1])
        assert st["err"] == 0 and st["nulls"] == 0 and st["sorted"] == 1
        assert st["nodes"] == len(np.unique(e))
        assert st["links"] == len(e)
        assert st["edge_xor"] == int(np.bitwise_xor.reduce(m))
        assert st["edge_sum"] == int(m.sum(dtype=np.uint64))
        assert st["lost_adds"] > 0  # threads raced to add the same key and the losers freed their node
        assert ins.check_canonical_empty(h.snapshot(), h.bitmaps()) == []
        assert h.error_flags() == 0


def _star(n):
    """n edges, most of them from one vertex: its queue is cut into many segments."""
    rng = np.random.default_rng(n)
    src = np.where(rng.random(n) < 0.8, 7, rng.integers(100, 140, n))
    return np.stack([src, rng.integers(1000, 1100, n)], 1).astype(np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("n,threads", [(1, 1), (128, 1), (129, 1), (3000, 1), (2, 2048), (3000, 2048), (40000, 2048)])
def test_gpu_graph_long_queue(n, threads):
    """A hot vertex's queue comes out whole and in order: one thread appends
    in edge order; many threads keep every source's sinks as a multiset."""
    from kma_b200 import Heap, graph
    from kma_b200 import inspect as ins
    e = _star(n)
    with Heap(2048, 14) as h:
        st, (keys, _, sinks, start) = graph.build(h, e, threads=threads, export=True)
        m = edge_mix(e[:, 0], e[:, 1])
        assert (st["links"], st["err"], st["nulls"], st["sorted"]) == (n, 0, 0, 1)
        assert st["edge_xor"] == int(np.bitwise_xor.reduce(m)) and st["edge_sum"] == int(m.sum(dtype=np.uint64))
        np.testing.assert_array_equal(keys, np.unique(e))
        for i, k in enumerate(keys):
            got, want = sinks[start[i]:start[i + 1]], e[e[:, 0] == k, 1].astype(np.int64)
            np.testing.assert_array_equal(*((got, want) if threads == 1 else (np.sort(got), np.sort(want))))
        assert ins.check_canonical_empty(h.snapshot(), h.bitmaps()) == []
        assert h.error_flags() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("edges,vertices,threads", [(2188, 547, 4096), (14928, 3732, 151552)])
def test_gpu_losers_of_inserts_give_their_blocks_back(edges, vertices, threads):
    """Small graphs by many threads: most inserts are lost, and the losers'
    per-thread frees, in divergent code, empty superblocks all the time.  No
    wait of the heap expires, and every superblock comes back."""
    from kma_b200 import Heap, graph
    from kma_b200 import inspect as ins
    e = graph.synth_edges(edges, edges, vertices)
    with Heap((1 << 30) >> 14, 14) as h:
        for _ in range(40):
            st, _ = graph.build(h, e, threads=threads, free_after=True)
            assert st["err"] == 0 and st["nulls"] == 0 and st["links"] == edges
            assert h.error_flags() == 0
        assert ins.check_canonical_empty(h.snapshot(), h.bitmaps()) == []
