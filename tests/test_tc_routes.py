"""Triangle counts of small graphs (bit rows, pairs of up neighbours) against the
DAG's tasks and the oracle, at the sizes where the route changes."""
import numpy as np
import pytest

from brute import random_graph
from conftest import csr_from_edges
from mercury_b200 import DeviceGraph, Graph, McError, tc_count_host
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def graphs():
    yield csr_from_edges(1, [])
    yield csr_from_edges(5, [])
    for n, p, seed in [(3, 1.0, 0), (31, 0.5, 1), (32, 1.0, 2), (33, 0.4, 3), (256, 0.05, 4),
                       (256, 0.2, 5), (257, 0.05, 6), (700, 0.02, 7)]:
        yield csr_from_edges(n, random_graph(n, p, seed))
    for n, mean, cap in [(1024, 12.0, 300.0), (1025, 12.0, 300.0), (20000, 13.0, 900.0),
                         (40000, 14.0, 90.0)]:
        g = Graph.chung_lu(n, 2.1, mean, cap, seed=n)
        yield np.array(g.rowptr), np.array(g.col)


@pytest.mark.parametrize("route", [None, "bits", "pairs", "dag"])
def test_routes_give_the_oracle_count(monkeypatch, route):
    """Each route, and the choice by size, on resident graphs and from host
    arrays; the DAG and the statistics are there after any of them."""
    if route:
        monkeypatch.setenv("MERCURY_TC_ROUTE", route)
    for rp, col in graphs():
        want = orc.tc(rp, col)
        with DeviceGraph(rp, col) as d:
            assert d.tc_count() == want
            drp, dcol = d.export_dag()
            wrp, wcol = orc.orient(rp, col)
            assert np.array_equal(drp, wrp) and np.array_equal(dcol, wcol)
            assert d.tc_stats()["dag_edges"] == len(col) // 2
            assert sum(d.tc_count_shard(s, 3) for s in range(3)) == want
            assert d.tc_count() == want
        assert tc_count_host(rp, col) == want


@pytest.mark.parametrize("n", [40, 3000])  # bit rows with their own checks; pairs
@pytest.mark.parametrize("fault", ["range", "negative", "order", "loop", "offsets", "ends"])
def test_small_host_graphs_are_checked(n, fault):
    g = Graph.chung_lu(n, 2.1, 6.0, 30.0, seed=2)
    rp, col = np.array(g.rowptr), np.array(g.col)
    row = int(np.argmax(np.diff(rp) >= 2))
    at = int(rp[row])
    if fault == "range":
        col[at + 1] = n
    elif fault == "negative":
        col[at] = -1
    elif fault == "order":
        col[at], col[at + 1] = col[at + 1], col[at]
    elif fault == "loop":
        col[at] = row
    elif fault == "offsets":
        rp[row + 1] = len(col) + 7
    else:
        rp[0] = 1
    with pytest.raises(McError):
        tc_count_host(rp, col)
    assert tc_count_host(g.rowptr, g.col) == orc.tc(g.rowptr, g.col)
