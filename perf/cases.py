"""Timed cases of the counting path: what a program that uses this package has
it do, through the package's public entry points.

Every input is made from the case and a seed on the GPU: RMAT draws
(quadrants 0.57, 0.19, 0.19, 0.05, no relabelling) and Chung-Lu draws
(weights (i + 1)^(-1 / (gamma - 1)) scaled to the mean degree, then capped),
the two families of the benchmark and the tests, with the duplicate pairs and
self-loops that raw edge lists have.  Counts are whole numbers, so every
output has one right value.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mercury_b200 import Batch, DeviceGraph, Graph, dgraph_from_edges, tc_count_host


def listed():
    return [
        # Resident graphs, counted again and again (mc_tc_count): one of the
        # smallest graphs of the batch and serving mixes, where launches and
        # host work are all there is; an ordinary one; the benchmark's.
        {"name": "tc_rmat8", "do": "tc", "graph": "rmat", "scale": 8, "edge_factor": 8},
        {"name": "tc_rmat16", "do": "tc", "graph": "rmat", "scale": 16, "edge_factor": 16},
        {"name": "tc_rmat22", "do": "tc", "graph": "rmat", "scale": 22, "edge_factor": 16},
        # The large graph of the serving mix: many short rows beside hubs of
        # degree above 10,000 (a social network's shape).
        {"name": "tc_powerlaw2m", "do": "tc", "graph": "chung_lu", "n": 2000000, "gamma": 2.1,
         "mean": 20.0, "cap": 50000.0},
        # The drop-in call of the reference's users (TCSolver): host arrays
        # in, count out, the copy to the device inside the call.
        {"name": "host_rmat20", "do": "tc_host", "graph": "rmat", "scale": 20, "edge_factor": 16},
        # A raw edge list already on the device, cleaned, built and counted.
        {"name": "edges_rmat20", "do": "edges", "graph": "rmat", "scale": 20, "edge_factor": 16},
        # The dataset step: a host edge list turned into CSR arrays.
        {"name": "convert_rmat16", "do": "convert", "graph": "rmat", "scale": 16,
         "edge_factor": 16},
        # All eight patterns of a small graph (the size of a batch's pattern
        # job), one call each, as a script over the `sm` programs does.
        {"name": "patterns_rmat8", "do": "patterns", "patterns": "12345678", "graph": "rmat",
         "scale": 8, "edge_factor": 8},
        # The pattern benchmark's graph: the tree patterns, then those that
        # hold a triangle.
        {"name": "trees_100k", "do": "patterns", "patterns": "1234", "graph": "chung_lu",
         "n": 100000, "gamma": 2.1, "mean": 10.0, "cap": 200.0},
        {"name": "cyclic_100k", "do": "patterns", "patterns": "5678", "graph": "chung_lu",
         "n": 100000, "gamma": 2.1, "mean": 10.0, "cap": 200.0},
        # A graph with hubs of degree above 4,096, on the patterns that
        # finish there.
        {"name": "hubs_60k", "do": "patterns", "patterns": "1478", "graph": "chung_lu",
         "n": 60000, "gamma": 2.1, "mean": 20.0, "cap": 50000.0},
        # The batched mode's mix: triangle jobs on RMAT scale 8 to max_scale,
        # P1..P8 on scale 5 to 8, one launch for all.
        {"name": "batch_512", "do": "batch", "graphs": 512, "max_scale": 14},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, max_pairs, min_pairs=500):
    """RMAT or Chung-Lu with a number of raw pairs between the two bounds."""
    pairs = _log_int(rng, min_pairs, max_pairs)
    if rng.random() < 0.4:
        ef = rng.choice([8, 16, 24, 32])
        scale = max(6, min(22, int(math.log2(pairs / ef))))
        return {"graph": "rmat", "scale": scale, "edge_factor": min(ef, max(2, pairs >> scale))}
    mean = round(rng.uniform(4, 32), 2)
    n = max(64, int(2 * pairs / mean)) | 1
    return {"graph": "chung_lu", "n": n, "gamma": rng.choice([2.1, 2.4, 3.0]), "mean": mean,
            "cap": float(rng.choice([100, 1000, 50000]))}


def draw(rng):
    do = rng.choice(["tc", "tc", "tc", "tc_host", "edges", "convert", "patterns", "patterns",
                     "hubs", "batch"])
    if do == "tc":
        return {"do": do, **_draw_graph(rng, 60_000_000)}
    if do == "tc_host":
        return {"do": do, **_draw_graph(rng, 16_000_000)}
    if do == "edges":
        return {"do": do, **_draw_graph(rng, 16_000_000)}
    if do == "convert":
        return {"do": do, **_draw_graph(rng, 4_000_000)}
    if do == "patterns":
        n = _log_int(rng, 200, 100_000) | 1
        return {"do": do, "patterns": rng.choice(["12345678", "1234", "5678", "1", "2", "3", "46"]),
                "graph": "chung_lu", "n": n, "gamma": rng.choice([2.1, 2.5]),
                "mean": round(rng.uniform(4, 10), 2), "cap": float(rng.randint(40, 200))}
    if do == "hubs":
        return {"do": "patterns", "patterns": rng.choice(["1478", "14", "78"]),
                "graph": "chung_lu", "n": _log_int(rng, 8_000, 60_000) | 1, "gamma": 2.1,
                "mean": round(rng.uniform(8, 20), 2), "cap": 50000.0}
    return {"do": "batch", "graphs": _log_int(rng, 16, 512), "max_scale": rng.randint(9, 14)}


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _pairs(case, seed):
    """(src, dst, n): int32 pairs on the GPU, duplicates and self-loops among them."""
    g, dev = _gen(seed), _device()
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        m = case["edge_factor"] * n
        src = torch.zeros(m, dtype=torch.int32, device=dev)
        dst = torch.zeros(m, dtype=torch.int32, device=dev)
        for _ in range(case["scale"]):
            r = torch.rand(m, device=dev, generator=g)
            lower = r >= 0.76
            right = ((r >= 0.57) & ~lower) | (r >= 0.95)
            src.mul_(2).add_(lower)
            dst.mul_(2).add_(right)
        return src, dst, n
    n = case["n"]
    m = int(n * case["mean"] / 2)
    w = torch.arange(1, n + 1, dtype=torch.float64, device=dev) ** (-1.0 / (case["gamma"] - 1.0))
    w = (w * (case["mean"] * n / w.sum())).clamp(max=case["cap"])
    total = torch.cumsum(w, 0)

    def ends():
        u = torch.rand(m, dtype=torch.float64, device=dev, generator=g) * total[-1]
        return torch.searchsorted(total, u).clamp(max=n - 1).to(torch.int32)

    return ends(), ends(), n


def _edge_file(case, seed):
    """The raw list up to its pair that brings the distinct edges to half of
    all pairs (a data set has a given number of edges)."""
    src, dst, n = _pairs(case, seed)
    a, b = src.long(), dst.long()
    at = torch.nonzero(a != b).flatten()
    key = (torch.minimum(a, b) * n + torch.maximum(a, b))[at]
    _, group = torch.unique(key, return_inverse=True)
    first = torch.full((int(group.max()) + 1,), src.numel(), dtype=torch.int64, device=src.device)
    first.scatter_reduce_(0, group, at, "amin")
    first = torch.sort(first).values
    stop = int(first[min(first.numel(), src.numel() // 2) - 1]) + 1
    return src[:stop], dst[:stop], n


def _sync():
    if torch.cuda.is_available():
        torch.cuda.synchronize()


def _resident(case, seed):
    src, dst, n = _pairs(case, seed)
    _sync()
    return dgraph_from_edges(src.data_ptr(), dst.data_ptr(), n, num_edges=src.numel(),
                             device_input=True)


def prepare(case, seed):
    do = case["do"]
    if do in ("tc", "patterns"):
        return {"do": do, "graph": _resident(case, seed),
                "patterns": [int(c) for c in case.get("patterns", "")]}
    if do == "tc_host":
        d = _resident(case, seed)
        rowptr, col = d.export_csr()
        d.close()
        return {"do": do, "rowptr": rowptr, "col": col}
    if do == "edges":
        src, dst, n = _pairs(case, seed)
        _sync()
        return {"do": do, "src": src, "dst": dst, "n": n}
    if do == "convert":
        src, dst, n = _edge_file(case, seed)
        return {"do": do, "src": src.cpu().numpy(), "dst": dst.cpu().numpy(), "n": n}
    rng = np.random.default_rng(seed)
    graphs, jobs = [], []
    for i in range(case["graphs"]):
        job = i % 9
        scale = int(rng.integers(8, case["max_scale"] + 1) if job == 0 else rng.integers(5, 9))
        ef = int(rng.integers(8, 33) if job == 0 else rng.integers(4, 9))
        graphs.append(Graph.rmat(scale, ef, seed=int(rng.integers(1, 1 << 40))))
        jobs.append(job)
    return {"do": do, "batch": Batch(graphs, jobs)}


def run(state):
    do = state["do"]
    if do == "tc":
        return state["graph"].tc_count()
    if do == "patterns":
        return [state["graph"].pattern_count(k) for k in state["patterns"]]
    if do == "tc_host":
        return tc_count_host(state["rowptr"], state["col"])
    if do == "edges":
        src, dst = state["src"], state["dst"]
        with dgraph_from_edges(src.data_ptr(), dst.data_ptr(), state["n"],
                               num_edges=src.numel(), device_input=True) as g:
            return {"triangles": g.tc_count(), "entries": g.nnz, "max_degree": g.max_degree}
    if do == "convert":
        with dgraph_from_edges(state["src"], state["dst"], state["n"]) as g:
            rowptr, col = g.export_csr()
        return {"rowptr": rowptr, "col": col}
    return state["batch"].count().astype(np.int64)


# ------------------------------------------------------------- the work done
def _size(case):
    """(vertices, raw pairs) of a case's graph."""
    if case["graph"] == "rmat":
        return 1 << case["scale"], case["edge_factor"] << case["scale"]
    return case["n"], int(case["n"] * case["mean"] / 2)


def work(case):
    """Bytes: the inputs read once (a CSR's int64 row offsets and int32
    columns, both directions; a pair's two ids), the outputs written once.
    Duplicate pairs are counted as entries.  Operations: one per entry read;
    what an intersection costs depends on the graph."""
    do = case["do"]
    if do == "batch":
        per_job = case["graphs"] / 9
        # Means over the uniform scales; edge factor 20 (triangles), 6 (patterns).
        tri = sum(2 * 20 * (1 << s) for s in range(8, case["max_scale"] + 1)) \
            / (case["max_scale"] - 7)
        pat = sum(2 * 6 * (1 << s) for s in range(5, 9)) / 4
        entries = per_job * (tri + 8 * pat)
        return {"bytes": 4.8 * entries + 8 * case["graphs"], "flops": entries}
    n, m = _size(case)
    csr = 8 * (n + 1) + 8 * m
    if do == "edges":
        return {"bytes": 8 * m + 8, "flops": 2 * m}
    if do == "convert":  # m / 2 distinct edges, each at least once in the list
        return {"bytes": 4 * m + 8 * (n + 1) + 4 * m, "flops": m}
    calls = len(case["patterns"]) if do == "patterns" else 1
    return {"bytes": calls * (csr + 8), "flops": calls * 2 * m}


def exact(case, seed):
    """The count or the CSR from plain torch, where that is quick: triangles
    as trace(A^3) / 6 up to 4,096 vertices, the CSR from sorted keys."""
    if case["do"] not in ("tc", "tc_host", "convert"):
        return None
    src, dst, n = (_edge_file if case["do"] == "convert" else _pairs)(case, seed)
    src, dst = src.long(), dst.long()
    keep = src != dst
    src, dst = src[keep], dst[keep]
    if case["do"] == "convert":
        key = torch.unique(torch.cat([src * n + dst, dst * n + src]))
        rows, col = key // n, key % n
        rowptr = torch.zeros(n + 1, dtype=torch.int64, device=key.device)
        rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
        return {"rowptr": rowptr.cpu().numpy(), "col": col.to(torch.int32).cpu().numpy()}
    if n > 4096:
        return None
    a = torch.zeros((n, n), dtype=torch.float64, device=src.device)
    a[src, dst] = 1.0
    a[dst, src] = 1.0
    return int(round(((a @ a) * a).sum().item())) // 6
