"""Pattern graphs of a batch at the ends of what the bit rows take: a batch of one
small dense graph, whose work goes in parts, and mixes of dense and sparse ones."""
import numpy as np
import pytest

from brute import random_graph
from conftest import csr_from_edges
from mercury_b200 import Batch, DeviceGraph, Graph

pytestmark = pytest.mark.gpu


def wants(rp, col):
    with DeviceGraph(rp, col) as d:
        return [d.tc_count()] + [d.pattern_count(k) for k in range(1, 9)]


@pytest.mark.parametrize("n,p", [(1, 0.0), (5, 1.0), (40, 1.0), (100, 1.0), (200, 0.5),
                                 (700, 0.01), (1000, 0.002), (1024, 0.05)])
def test_a_batch_of_one_graph(n, p):
    rp, col = csr_from_edges(n, random_graph(n, p, n))
    want = wants(rp, col)
    for job in range(9):
        with Batch([Graph.from_csr(rp, col)], [job]) as b:
            assert b.count().tolist() == [want[job]]


@pytest.mark.parametrize("route", ["default", "dense", "formula"])
def test_dense_and_sparse_graphs_in_one_batch(monkeypatch, route):
    arrays = [csr_from_edges(n, random_graph(n, p, n)) for n, p in
              [(60, 1.0), (60, 0.1), (300, 0.9), (900, 0.003), (1000, 0.05), (1030, 0.01)]]
    graphs, jobs, want = [], [], []
    for rp, col in arrays:
        graphs += [Graph.from_csr(rp, col)] * 9
        jobs += list(range(9))
        want += wants(rp, col)
    if route != "default":
        monkeypatch.setenv("MERCURY_MOTIF_ROUTE", route)
    with Batch(graphs, jobs) as b:
        assert b.count().tolist() == want


def test_a_lone_graph_does_not_wait_for_one_cta():
    """P5 of one complete graph of 100 vertices: 5.3 ms on a single CTA, 0.6 ms by
    the per-edge formulas."""
    i, j = np.tril_indices(100, -1)
    rp, col = csr_from_edges(100, np.stack([i, j], 1))
    with Batch([Graph.from_csr(rp, col)], [5]) as b:
        b.count()
        best = min(b.count() is not None and b.last_timing.count_ms for _ in range(10))
    assert best < 2.0


def test_sparse_graphs_do_not_wait_for_all_pairs():
    """P4 of 40 paths of 1,000 vertices: 1.15 ms with every pair's rows, 0.12 ms by
    the per-edge formulas."""
    a = np.arange(999)
    rp, col = csr_from_edges(1000, np.stack([a, a + 1], 1))
    with Batch([Graph.from_csr(rp, col)] * 40, [4] * 40) as b:
        b.count()
        best = min(b.count() is not None and b.last_timing.count_ms for _ in range(10))
    assert best < 0.5
