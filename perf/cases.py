"""The measured work of kma_b200: what a user of the framework has it do,
through the package's public entry points.

Six kinds, each with a range of its own:

  wl      the stress programs on a KMA heap (`Workload`): config 1 through
          begin / rounds / stats, config 2 end to end through `run_host`
          (pinned host seeds in, per-item hashes and counters out)
  batch   many uneven jobs in one captured launch (`Batch`), on a KMA heap or
          on the PMA bump heap, with and without the per-warp cache
  serve   requests served over one resident heap (`Server.run`)
  queue   one queue, or many, filled and emptied by many threads
          (`structs.c3_queue`): per thread, warp or block calls
  tree    concurrent insert / lookup / remove (`structs.c3_tree`)
  graph   the graph build over tree, queues and heap (`graph.build`), with
          the teardown or with the export of the graph

Every output is a whole number (counters, checksums, results per operation,
keys): none is rounded, so there is no 64-bit value to compare with.  Not
returned, because two runs of one build differ in them: block offsets and
what is hashed from them, the order of links in a concurrent build, lost
races, cache hits, and measured times.

Heaps are sized so that no request fails for want of room; a failing one
would make the counters depend on the order of the threads.
"""
import math

import numpy as np
import torch

from kma_b200 import MODE_PLAIN, MODE_WARP, WL_C1, WL_C2, Heap, Workload, graph, structs
from kma_b200.batch import Batch
from kma_b200.serve import STATUS, Server

MODES = {"plain": MODE_PLAIN, "warp": MODE_WARP}
QKINDS = {"clqueue": structs.C3_CLQUEUE, "iqueue": structs.C3_IQUEUE}
QFORMS = {"thread": 0, "warp": structs.C3_WARP, "block": structs.C3_BLOCK}
C2_MEAN = sum(8 << k for k in range(9)) / 9
C1_MEAN = (8 + 16 + 32 + 64 + 128 + 256) / 6
# Zipf(1.2) over the 512 multiples of 8 up to 4096: mean request of the jobs
ZIPF_MEAN = sum(8 * k * k ** -1.2 for k in range(1, 513)) / sum(k ** -1.2 for k in range(1, 513))


def listed():
    return [
        # the smallest program: 4 work-groups of 64, a 16 MiB heap of 4 KiB superblocks; launches and
        # round trips count
        {"name": "c1_256_items", "kind": "wl", "program": 1, "mode": "warp", "items": 256, "rounds": 16,
         "sb_log2": 12, "heap_mib": 16, "block_dim": 64},
        # the reference's own calls, one malloc / free per thread, at an odd size that leaves half of the GPU idle
        {"name": "c2_plain_50021", "kind": "wl", "program": 2, "mode": "plain", "items": 50021, "rounds": 32,
         "sb_log2": 14, "heap_mib": 1024, "block_dim": 0},
        # the headline: full occupancy, 64 rounds, fragmentation building up, end to end from host buffers
        {"name": "c2_warp_303104", "kind": "wl", "program": 2, "mode": "warp", "items": 303104, "rounds": 64,
         "sb_log2": 14, "heap_mib": 1024, "block_dim": 0},
        # a few small, ragged jobs (one of 5 threads) in one graph launch
        {"name": "batch_8_jobs", "kind": "batch", "heap": "kma", "jobs": 8, "lo": 5, "hi": 40000, "rounds": 12,
         "mode": "warp", "sb_log2": 14, "heap_mib": 512, "block_dim": 256, "cache": 0},
        # the batched configuration's heap and geometry: 64 jobs from 1k threads up, per-warp caches
        {"name": "batch_64_jobs", "kind": "batch", "heap": "kma", "jobs": 64, "lo": 1000, "hi": 400000, "rounds": 16,
         "mode": "warp", "sb_log2": 14, "heap_mib": 16384, "block_dim": 256, "cache": 4},
        # the same program composed with the bump heap
        {"name": "batch_pma_24_jobs", "kind": "batch", "heap": "pma", "jobs": 24, "lo": 1000, "hi": 200000,
         "rounds": 16, "mode": "warp", "sb_log2": 0, "heap_mib": 16384, "block_dim": 256, "cache": 0},
        # a server under full load: every request is there, 16 slots, sizes over the served range
        {"name": "serve_burst_64", "kind": "serve", "requests": 64, "nmin": 1000, "nmax": 1000000, "slots": 16,
         "mode": "warp", "sb_log2": 14, "heap_mib": 8192},
        # one hot FIFO between 2^18 producers and consumers
        {"name": "clqueue_block_4m", "kind": "queue", "queue": "clqueue", "form": "block", "threads": 1 << 18,
         "per_thread": 16, "shards": 1},
        # the indexed queue spread over shards, plain calls per thread, 2^24 payloads
        {"name": "iqueue_shards_16m", "kind": "queue", "queue": "iqueue", "form": "thread", "threads": 1 << 18,
         "per_thread": 64, "shards": 4096},
        # the tree at half its configuration's size, mixed 50/30/20
        {"name": "tree_2m_ops", "kind": "tree", "ops": 1 << 21, "threads": 1 << 18},
        # a skewed graph: one vertex owns a large share of all edges; built, checked and torn down
        {"name": "graph_zipf_1m", "kind": "graph", "edges": 1 << 20, "vertices": 1 << 18, "skew": 1.1,
         "threads": 148 * 1024, "heap": "kma", "heap_mib": 1024, "export": False},
        # a small ordinary graph that the caller reads back
        {"name": "graph_export_200k", "kind": "graph", "edges": 200000, "vertices": 20000, "skew": 0.6,
         "threads": 65536, "heap": "kma", "heap_mib": 256, "export": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wl", "wl", "batch", "batch", "serve", "queue", "queue", "tree", "graph"])
    if kind == "wl":
        program = rng.choice([1, 2, 2])
        items = _log(rng, 200, 300000)
        # room for the live blocks of every item and for the superblocks that the classes hold
        heap = max(64, items * 8 >> 10) if program == 2 else max(16, items >> 9)
        return {"kind": kind, "program": program, "mode": rng.choice(["plain", "warp", "warp"]), "items": items,
                "rounds": rng.randint(4, 64), "sb_log2": rng.choice([12, 14]), "heap_mib": heap,
                "block_dim": rng.choice([0, 64, 128, 256])}
    if kind == "batch":
        heap = rng.choice(["kma", "kma", "pma"])
        hi = _log(rng, 2000, 300000)
        mode = rng.choice(["plain", "warp", "warp", "warp"])
        jobs = rng.randint(3, 32)
        return {"kind": kind, "heap": heap, "jobs": jobs, "lo": rng.choice([5, 1000]), "hi": hi,
                "rounds": rng.randint(4, 16), "mode": mode, "sb_log2": 14 if heap == "kma" else 0,
                "heap_mib": 16384 if jobs * hi > 1000000 else 4096, "block_dim": rng.choice([128, 256, 512]),
                "cache": rng.choice([0, 2, 4]) if heap == "kma" and mode == "warp" else 0}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(1, 64), "nmin": 1000, "nmax": _log(rng, 10000, 600000),
                "slots": rng.choice([1, 4, 8, 16]), "mode": rng.choice(["plain", "warp", "warp"]), "sb_log2": 14,
                "heap_mib": 8192}
    if kind == "queue":
        form = rng.choice(["thread", "warp", "block"])
        queue = rng.choice(["clqueue", "iqueue"])
        shards = 1 if form == "block" else rng.choice([1, 64, 1024, 4096])
        # one queue serves a few million calls a second when each thread calls for itself
        most = {"thread": 16, "warp": 20, "block": 21}[form] if shards == 1 else 23
        per = rng.choice([1, 7, 16, 64])
        threads = max(1, _log(rng, 1000, 1 << most) // per)
        return {"kind": kind, "queue": queue, "form": form, "threads": threads, "per_thread": per, "shards": shards}
    if kind == "tree":
        ops = _log(rng, 1000, 1500000)
        return {"kind": kind, "ops": ops, "threads": max(1, ops // rng.choice([4, 16]))}
    edges = _log(rng, 2000, 700000)
    heap = rng.choice(["kma", "kma", "pma"])
    return {"kind": kind, "edges": edges, "vertices": max(100, edges // rng.choice([4, 10])),
            "skew": rng.choice([0.0, 0.6, 1.1]), "threads": rng.choice([4096, 65536, 148 * 1024]), "heap": heap,
            "heap_mib": 1024, "export": rng.random() < 0.4}


def _rng(case, seed):
    return np.random.default_rng([0x4B4D41, seed])


def _heap(case):
    return Heap((case["heap_mib"] << 20) >> case.get("sb_log2", 14), case.get("sb_log2", 14))


def _edges(g, n_edges, n_vertices, skew):
    """(source, sink) pairs over random distinct u32 keys: both ends by rank Zipf(skew), and one edge more
    from every vertex, so that each is in the graph."""
    keys = g.choice(2**32 - 1, size=n_vertices, replace=False).astype(np.uint32)
    p = np.arange(1, n_vertices + 1, dtype=np.float64) ** -skew
    ends = g.choice(n_vertices, size=(n_edges, 2), p=p / p.sum())
    ends[g.permutation(n_edges)[:n_vertices], 0] = np.arange(n_vertices)
    return keys[ends]


def prepare(case, seed):
    g = _rng(case, seed)
    kind = case["kind"]
    if kind == "wl":
        heap = _heap(case)
        w = Workload(heap, WL_C1 if case["program"] == 1 else WL_C2, case["items"])
        s = {"heap": heap, "wl": w, "seed": int(g.integers(1, 1 << 62))}
        if case["program"] == 2:
            ids = np.arange(case["items"], dtype=np.uint64)
            seeds = np.uint64(s["seed"]) ^ (ids * np.uint64(0x9E3779B97F4A7C15))
            s["seeds"] = torch.from_numpy(seeds.view(np.int64)).pin_memory()
            s["hashes"] = torch.empty(case["items"], dtype=torch.int64).pin_memory()
    elif kind == "batch":
        # thread counts spread log-uniformly, one of each stratum so that the total does not hang on one draw
        u = (np.arange(case["jobs"]) + g.random(case["jobs"])) / case["jobs"]
        threads = np.exp(np.log(case["lo"]) + u * np.log(case["hi"] / case["lo"])).astype(np.int64)
        heap = structs.Pma(case["heap_mib"] << 20) if case["heap"] == "pma" else _heap(case)
        b = Batch(heap, g.permutation(threads), g.integers(0, 2**63, case["jobs"]), case["rounds"],
                  mode=MODES[case["mode"]])
        stream = torch.cuda.Stream()
        b.capture(case["block_dim"], case["cache"], stream)
        s = {"heap": heap, "batch": b, "stream": stream}
    elif kind == "serve":
        n = case["requests"]
        u = (np.arange(n) + g.random(n)) / n
        nv = np.exp(np.log(case["nmin"]) + u * np.log(case["nmax"] / case["nmin"])).astype(np.int64)
        heap = _heap(case)
        s = {"heap": heap, "server": Server(heap, slots=case["slots"], max_vertices=1_000_000,
                                            mode=MODES[case["mode"]]),
             "nv": g.permutation(nv), "seeds": g.integers(0, 2**63, n)}
    elif kind == "queue":
        # how many producers there are changes from run to run
        threads = case["threads"] + int(g.integers(0, max(64, case["threads"] // 64)))
        s = {"seed": int(g.integers(1, 1 << 62)), "threads": threads}
    elif kind == "tree":
        s = {"kinds": g.choice(3, size=case["ops"], p=(0.5, 0.3, 0.2)).astype(np.uint8),
             # a key drawn twice or more is what lookups and removes find
             "keys": g.integers(0, 1 << 32, size=max(1, case["ops"] // 2), dtype=np.uint64).astype(np.uint32)[
                 g.integers(0, max(1, case["ops"] // 2), size=case["ops"])]}
    else:
        edges = _edges(g, case["edges"], case["vertices"], case["skew"])
        heap = structs.Pma(case["heap_mib"] << 20) if case["heap"] == "pma" else _heap(case)
        s = {"heap": heap, "edges": edges}
    s["case"] = case
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "wl":
        mode = MODES[case["mode"]]
        if case["program"] == 1:
            s["heap"].reset()
            s["wl"].begin(s["seed"])
            s["wl"].rounds(case["rounds"], mode, block_dim=case["block_dim"])
            st = s["wl"].stats()
        else:
            st = s["wl"].run_host(s["seeds"].data_ptr(), case["rounds"], mode, s["hashes"].data_ptr())
        return {k: st[k] for k in ("mallocs", "frees", "nulls", "bad_tags", "fill_bytes", "verify_bytes")}
    if kind == "batch":
        s["batch"].launch(s["stream"])
        st = s["batch"].stats(s["stream"])
        return {k: st[k] for k in ("mallocs", "frees", "nulls", "bad_tags", "fill_bytes", "verify_bytes", "retired",
                                   "refused")}
    if kind == "serve":
        res, summary = s["server"].run(s["nv"], s["seeds"])
        words = list(STATUS.values())
        out = {k: np.array([r[k] for r in res], np.uint64).view(np.int64)
               for k in ("checksum", "edges", "mallocs", "frees", "nulls")}
        return dict(out, status=np.array([words.index(r["status"]) for r in res]), ops=summary["ops"])
    if kind == "queue":
        st = structs.c3_queue(QKINDS[case["queue"]] | QFORMS[case["form"]], s["threads"], case["per_thread"],
                              case["shards"], seed=s["seed"])
        return {k: st[k] for k in ("enqueued", "dequeued", "empty", "remaining", "out_count", "out_xor", "out_sum",
                                   "in_xor", "in_sum", "err", "walk_ok")}
    if kind == "tree":
        res, st = structs.c3_tree(s["kinds"], s["keys"], case["threads"])
        return res, {k: st[k] for k in ("live_keys", "keys_xor", "keys_sum", "sorted", "err")}
    if case["heap"] == "pma":
        s["heap"].reset()
    st, exported = graph.build(s["heap"], s["edges"], case["threads"], free_after=True, export=case["export"])
    out = {k: st[k] if st[k] < 1 << 63 else st[k] - (1 << 64)
           for k in ("nodes", "links", "nulls", "edge_xor", "edge_sum", "sorted", "err")}
    if exported is not None:
        out["keys"], out["link_start"] = exported[0], exported[3]
    return out


def work(case):
    """Payload written and read once, and each structure's own words once."""
    kind = case["kind"]
    if kind == "wl":
        n = case["items"] * case["rounds"]
        mean = C1_MEAN if case["program"] == 1 else C2_MEAN
        return {"bytes": 2.0 * n * mean, "flops": 0}
    if kind == "batch":
        # mean of a log-uniform thread count
        threads = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": 2.0 * case["jobs"] * threads * case["rounds"] * ZIPF_MEAN, "flops": 0}
    if kind == "serve":
        verts = case["requests"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        # ids written and read once (mean degree of d^-2.1 on 1..4096: 3.6) and a page header and list per vertex
        return {"bytes": verts * (2 * 4 * 3.6 + 2 * 24 + 48), "flops": 0}
    if kind == "queue":
        # 16-byte items written when appended, read when taken
        return {"bytes": 32.0 * case["threads"] * case["per_thread"], "flops": 0}
    if kind == "tree":
        # kind, key and result of each operation; a 24-byte node of each of the (about 0.43) inserted keys, read once more
        return {"bytes": case["ops"] * 6.0 + 2 * 24.0 * 0.32 * case["ops"], "flops": 0}
    # the edge, its link written and read, and the nodes
    return {"bytes": case["edges"] * (8.0 + 2 * 16) + case["vertices"] * 2 * 40.0, "flops": 0}
