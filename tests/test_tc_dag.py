"""Whole triangle counts over the DAG's tasks (hub and leaf kernels) on graphs that
the default route counts otherwise, and every route's golden counts."""
import json
import os

import numpy as np
import pytest

from conftest import GOLDEN
from mercury_b200 import DeviceGraph, Graph, tc_count_host
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

with open(os.path.join(GOLDEN, "golden.json")) as f:
    GOLD = json.load(f)


@pytest.mark.parametrize("route", ["dag", "pairs", "bits"])
@pytest.mark.parametrize("name", sorted(GOLD))
def test_golden_counts_by_route(monkeypatch, name, route):
    monkeypatch.setenv("MERCURY_TC_ROUTE", route)
    g = Graph(os.path.join(GOLDEN, "graphs", name, "graph"))
    with DeviceGraph(g) as d:
        assert [d.tc_count() for _ in range(2)] == [GOLD[name]["TC"]] * 2
    assert tc_count_host(g.rowptr, g.col) == GOLD[name]["TC"]


def test_a_setting_of_the_kernels_keeps_the_dag_and_no_other_name_does(monkeypatch):
    """Small graphs are counted without the DAG unless a setting asks for a form of
    its kernels; a name that no kernel reads changes nothing."""
    g = Graph.rmat(10, 16, seed=2)
    want = orc.tc(g.rowptr, g.col)
    with DeviceGraph(g) as d:
        assert d.tc_count() == want
        small = d.last_timing.launches
        monkeypatch.setenv("MERCURY_DAG_STAGE", "0")
        assert d.tc_count() == want and d.last_timing.launches == small
        monkeypatch.setenv("MERCURY_TC_SHORT_RANGES", "0")
        assert d.tc_count() == want and d.last_timing.launches > small


@pytest.mark.parametrize("n,cap", [(2000, 300.0), (20000, 2000.0)])
def test_dag_counts_below_and_above_the_leaf_limit(monkeypatch, n, cap):
    """Graphs whose bound on d+ rules out hub tasks, and one with both kinds, from the
    bound alone (no wait) and through host arrays (with one)."""
    monkeypatch.setenv("MERCURY_TC_ROUTE", "dag")
    g = Graph.chung_lu(n, 2.1, 12.0, cap, seed=n)
    rp, col = np.array(g.rowptr), np.array(g.col)
    want = orc.tc(rp, col)
    with DeviceGraph(rp, col) as d:
        assert d.tc_count() == want
        assert sum(d.tc_count_shard(i, 2) for i in range(2)) == want
    with DeviceGraph(rp, col, host_columns=True) as d:
        assert d.tc_count() == want
    assert tc_count_host(rp, col) == want
