"""P1..P8 from motif sums (mercury_b200/csrc/motifs.cu).

CPU: the identities themselves -- every pattern as a signed combination of
sums over vertices, edges, triangles and vertex pairs -- restated in Python
and checked against the oracle's counts.  GPU: the route at the sizes where
its stages change form, against the oracle and against the formula routes.
"""
import math

import numpy as np
import pytest

from brute import random_graph
from conftest import csr_from_edges
from mercury_b200 import Batch, DeviceGraph, Graph
from oracle import oracle as orc


def motif_sums(rp, col):
    n = len(rp) - 1
    N = [set(int(x) for x in col[rp[v]:rp[v + 1]]) for v in range(n)]
    d = [len(s) for s in N]
    a = {(u, v): len(N[u] & N[v]) for u in range(n) for v in N[u]}
    t = [sum(a[v, x] for x in N[v]) // 2 for v in range(n)]
    d2 = [sum(d[p] - 1 for p in N[v]) for v in range(n)]
    C = math.comb
    s = dict.fromkeys("d3 d4 t2 td D C3 p4 fork dart T cricket bull lolli kite gem kd ka kk "
                      "K4 K5 C4 C4d C4a X7 W4 K23".split(), 0)
    for v in range(n):
        s["d3"] += C(d[v], 3)
        s["d4"] += C(d[v], 4)
        s["t2"] += C(t[v], 2)
        s["td"] += t[v] * d[v]
    for (u, v), x in a.items():
        if u > v:
            continue
        s["D"] += C(x, 2)
        s["C3"] += C(x, 3)
        s["p4"] += (d[u] - 1 - x) * (d[v] - 1 - x)
        s["fork"] += (C(d[u] - 1, 2) * (d[v] - 1) + C(d[v] - 1, 2) * (d[u] - 1)
                      - x * (d[u] + d[v] - 4))
        s["dart"] += C(x, 2) * (d[u] + d[v] - 6)
        for z in (N[u] & N[v]):
            if z < v:
                continue
            S = N[u] & N[v] & N[z]
            k = len(S)
            dd, aa = (d[u], d[v], d[z]), (a[v, z], a[u, z], a[u, v])  # aa[i] opposite dd[i]
            s["T"] += 1
            s["cricket"] += sum(C(q - 2, 2) for q in dd)
            s["bull"] += sum((dd[i] - 2) * (dd[i - 1] - 2) for i in range(3)) - sum(aa) + 3
            s["lolli"] += d2[u] + d2[v] + d2[z] - 2 * (sum(dd) - 3) - 2 * (sum(aa) - 3)
            s["kite"] += sum((aa[i] - 1) * (dd[i] - 2) for i in range(3))
            s["gem"] += sum((aa[i] - 1) * (aa[i - 1] - 1) for i in range(3))
            s["kd"] += k * sum(dd)
            s["ka"] += k * sum(aa)
            s["kk"] += C(k, 2)
            for w in (x for x in S if x > z):
                s["K4"] += 1
                s["K5"] += sum(1 for y in S & N[w] if y > w)
    for x in range(n):
        for y in range(x):
            S = N[x] & N[y]
            c = len(S)
            s["C4"] += C(c, 2)  # twice the 4-cycles, as are C4d and C4a
            s["K23"] += C(c, 3)
            s["C4d"] += C(c, 2) * (d[x] + d[y]) + sum((c - 1) * d[v] for v in S)
            s["C4a"] += sum((c - 1) * (a[x, v] + a[v, y]) for v in S)
            s["X7"] += sum((c - 2) * len(N[p] & S) for p in S)
            s["W4"] += sum(C(len(N[v] & S), 2) for v in S)
    s["X7"] //= 2
    s["W4"] //= 2
    return s


def counts(s):
    ka, kd = s["ka"] - 24 * s["K4"], s["kd"] - 36 * s["K4"]
    gem, kite = s["gem"] - 12 * s["K4"], s["kite"] - 12 * s["K4"]
    claw = s["d3"] - s["td"] + 6 * s["T"] + 2 * s["D"] - 4 * s["K4"]
    butterfly = s["t2"] - 2 * s["D"]
    house2, banner2 = s["C4a"] - 8 * s["D"], s["C4d"] - 8 * s["C4"] - 4 * s["D"]
    paw = s["td"] - 6 * s["T"] - 4 * (s["D"] - 6 * s["K4"]) - 12 * s["K4"]
    star = (s["d4"] - s["cricket"] + s["dart"] + butterfly - gem + s["W4"] - kd // 3 + ka
            - 2 * s["C3"] - 3 * s["kk"] + 5 * s["K5"])
    return [
        claw,
        s["fork"] - 2 * s["cricket"] - 2 * s["bull"] - s["lolli"] - banner2 + 6 * s["K23"]
        + 5 * s["dart"] + 4 * kite + 2 * house2 + 4 * butterfly - 10 * gem - 10 * s["X7"]
        + 20 * s["W4"] - 3 * kd + 10 * ka - 12 * s["C3"] - 36 * s["kk"] + 60 * s["K5"],
        4 * star + 3 * claw,
        s["p4"] - 2 * s["C4"] + 4 * s["D"] - 12 * s["K4"],
        2 * s["bull"] - 4 * s["dart"] - 4 * kite - house2 + 10 * gem + 8 * s["X7"] - 24 * s["W4"]
        + 4 * kd - 14 * ka + 12 * s["C3"] + 60 * s["kk"] - 120 * s["K5"],
        2 * paw + 2 * s["dart"] - 4 * gem + 8 * s["W4"] - 2 * kd + 10 * ka - 12 * s["C3"]
        - 48 * s["kk"] + 120 * s["K5"],
        2 * s["C3"] - ka + 6 * s["kk"] - 20 * s["K5"],
        kd - 3 * ka + 18 * s["kk"] - 60 * s["K5"],
    ]


@pytest.mark.parametrize("n,p,seed", [(6, 1.0, 0), (12, 0.3, 1), (16, 0.5, 2), (14, 0.8, 3),
                                      (25, 0.6, 4), (40, 0.1, 5), (30, 0.25, 6)])
def test_identities_give_the_oracle_counts(n, p, seed):
    rp, col = csr_from_edges(n, random_graph(n, p, seed))
    assert counts(motif_sums(rp, col)) == [orc.pattern(rp, col, k) for k in range(1, 9)]


def gpu_counts(rp, col):
    with DeviceGraph(rp, col) as d:
        return [d.pattern_count(k) for k in range(1, 9)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,seed", [
    (1, 0.0, 0), (2, 1.0, 0), (3, 1.0, 0), (4, 1.0, 0), (5, 1.0, 0), (6, 0.0, 0),
    (31, 0.4, 5), (32, 0.4, 5),    # bit rows of one whole word and a part
    (33, 1.0, 0), (34, 1.0, 0),    # d+ of 32 (one warp's rows) and of 33
    (64, 0.3, 6), (65, 1.0, 0), (70, 0.9, 1), (100, 0.3, 2), (180, 0.5, 3), (300, 0.02, 4)])
@pytest.mark.parametrize("route", ["default", "dense", "sparse"])
def test_motif_routes_vs_oracle(monkeypatch, n, p, seed, route):
    if route != "default":
        monkeypatch.setenv("MERCURY_MOTIF_ROUTE", route)
    rp, col = csr_from_edges(n, random_graph(n, p, seed))
    assert gpu_counts(rp, col) == [orc.pattern(rp, col, k) for k in range(1, 9)]


@pytest.mark.gpu
@pytest.mark.parametrize("make", [
    # Pair tables of every class (walks below 512 to above 32,768), degrees on
    # both sides of 512; tables over all vertices in shared memory.
    lambda: Graph.chung_lu(30001, 2.1, 12.0, 900.0, seed=7),
    # More vertices than the shared tables hold.
    lambda: Graph.chung_lu(150001, 2.1, 6.0, 3000.0, seed=3),
    lambda: Graph.rmat(11, 16, seed=5),
    # The largest graphs the bit rows take.
    lambda: Graph.chung_lu(1024, 2.1, 12.0, 300.0, seed=5),
], ids=["classes", "global_tables", "rmat11", "n1024"])
def test_motif_route_equals_formula_routes(monkeypatch, make):
    g = make()
    monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "sparse")
    with DeviceGraph(g) as d:
        motif = [d.pattern_count(k) for k in range(1, 9)]
        if g.n <= 1024:
            monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "dense")
            assert motif == [d.pattern_count(k) for k in range(1, 9)]
        monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "formula")
        assert motif == [d.pattern_count(k) for k in range(1, 9)]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [300, 700, 1200])
def test_motif_route_on_a_clique_with_a_tail(monkeypatch, n):
    """A clique of n with one vertex hung on vertex 0 holds C(n - 1, 2)
    induced paws and C(n - 1, 3) induced tailed K4s, and none of the other
    subgraphs.  At 700 the common-neighbour lists outgrow the first guess
    (64 M entries): the count starts over with the room asked for; at 1,200
    that is above 512 M entries, and a counting pass sizes them."""
    monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "sparse")
    i, j = np.tril_indices(n, -1)
    edges = np.stack([np.concatenate([i, [0]]), np.concatenate([j, [n]])], axis=1)
    adj = np.zeros((n + 1, n + 1), dtype=bool)
    adj[edges[:, 0], edges[:, 1]] = adj[edges[:, 1], edges[:, 0]] = True
    rp = np.concatenate([[0], np.cumsum(adj.sum(axis=1))]).astype(np.int64)
    col = np.nonzero(adj)[1].astype(np.int32)
    patterns = range(1, 9) if n == 300 else (1, 8)
    want = [0] * 8
    want[5], want[7] = 2 * math.comb(n - 1, 2), 3 * math.comb(n - 1, 3)
    with DeviceGraph(rp, col) as d:
        assert [d.pattern_count(k) for k in patterns] == [want[k - 1] for k in patterns]


@pytest.mark.gpu
def test_batch_bit_rows_at_word_edges(monkeypatch):
    """Every pattern of graphs at the edges of the bit rows' words and of
    their largest size (1,024 vertices), beside a triangle job and a larger
    pattern graph: the batch's counts are the formula routes'."""
    sizes = [1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 700, 1024, 1025]
    graphs, jobs = [], []
    for i, n in enumerate(sizes):
        g = (Graph.chung_lu(n, 2.1, 8.0, 60.0, seed=i + 1) if n > 8 else
             Graph.from_csr(*csr_from_edges(n, random_graph(n, 1.0, i))))
        graphs += [g] * 9
        jobs += list(range(9))
    with Batch(graphs, jobs) as b:
        got = b.count().tolist()
        b.autotune()
        assert b.count().tolist() == got
    monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "formula")
    want = []
    for g in graphs[::9]:
        with DeviceGraph(g) as d:
            want += [d.tc_count()] + [d.pattern_count(k) for k in range(1, 9)]
    assert got == want


@pytest.mark.gpu
@pytest.mark.parametrize("n,cap,ids", [(5000, 5000.0, "hubs first"), (12000, 12000.0, "hubs last"),
                                       (12000, 12000.0, "shuffled")])
def test_walks_in_parts(n, cap, ids):
    """Hubs whose walks outlast an SM's share of all walks (ordered pairs, in
    parts of the table's range), with the hubs at either end of the ids, isolated
    vertices at both, and shuffled."""
    g = Graph.chung_lu(n, 2.1, 30.0, cap, seed=n)
    rp, col = np.array(g.rowptr), np.array(g.col)
    src = np.repeat(np.arange(n), np.diff(rp))
    perm = {"hubs first": np.arange(n), "hubs last": np.arange(n)[::-1],
            "shuffled": np.random.default_rng(n).permutation(n)}[ids]
    keep = src < col
    rp, col = csr_from_edges(n + 20, np.stack([perm[src[keep]] + 7, perm[col[keep]] + 7], 1))
    with DeviceGraph(rp, col) as d:
        assert d.pattern_count(4) == orc.pattern_fast(rp, col, 4)
