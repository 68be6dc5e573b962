"""Bounded waits of the chained scans (task lists, radix passes) that give up:
every call that depends on them fails with an error, none of its kernels uses
what was left unwritten, and the next call on the same handle is right."""
import numpy as np
import pytest

from mercury_b200 import Batch, DeviceGraph, Graph, McError, dgraph_from_edges, tc_count_host
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    """Several blocks of task lists and several tiles of the rank sort."""
    g = Graph.rmat(14, 16, seed=3)
    rp, col = np.array(g.rowptr), np.array(g.col)
    return rp, col, orc.tc(rp, col)


def fails_then_counts(monkeypatch, call, want):
    assert call() == want
    monkeypatch.setenv("MERCURY_WAIT_POLLS", "0")
    for _ in range(2):
        with pytest.raises(McError, match="error flag"):
            call()
    monkeypatch.delenv("MERCURY_WAIT_POLLS")
    assert call() == want


def test_resident_and_one_shot_counts(monkeypatch, graph):
    rp, col, want = graph
    monkeypatch.setenv("MERCURY_TC_ROUTE", "dag")
    with DeviceGraph(rp, col) as d:
        fails_then_counts(monkeypatch, d.tc_count, want)
        fails_then_counts(monkeypatch, lambda: sum(d.tc_count_shard(i, 3) for i in range(3)), want)
    fails_then_counts(monkeypatch, lambda: tc_count_host(rp, col), want)


def test_a_failed_dag_is_built_again(monkeypatch):
    """tc_stats and export_dag after a count without the DAG build it; one that
    failed is not taken for a built one."""
    g = Graph.rmat(13, 16, seed=3)  # small enough for the pairs
    rp, col = np.array(g.rowptr), np.array(g.col)
    want = orc.tc(rp, col)
    monkeypatch.setenv("MERCURY_TC_ROUTE", "pairs")
    wrp, wcol = orc.orient(rp, col)
    with DeviceGraph(rp, col) as d:
        assert d.tc_count() == want
        monkeypatch.setenv("MERCURY_WAIT_POLLS", "0")
        for _ in range(2):
            with pytest.raises(McError, match="error flag"):
                d.tc_stats()
            with pytest.raises(McError, match="error flag"):
                d.export_dag()
        monkeypatch.delenv("MERCURY_WAIT_POLLS")
        drp, dcol = d.export_dag()
        assert np.array_equal(drp, wrp) and np.array_equal(dcol, wcol)


def test_batch_labels_cliques_and_builds(monkeypatch, graph):
    rp, col, want = graph
    monkeypatch.setenv("MERCURY_WAIT_POLLS", "0")
    with Batch([Graph.from_csr(rp, col)], [0]) as b:
        with pytest.raises(McError, match="error flag"):
            b.count()
    monkeypatch.setenv("MERCURY_CLIQUE_ROUTE", "cliques")
    with DeviceGraph(rp, col) as d:
        d.set_vlabels(np.zeros(len(rp) - 1, dtype=np.uint8), 0)
        for call in (lambda: d.pattern_count(7), d.tc_count_by_label):
            with pytest.raises(McError, match="error flag"):
                call()
        monkeypatch.delenv("MERCURY_WAIT_POLLS")
        assert int(d.tc_count_by_label()[0]) == want
    src = np.repeat(np.arange(len(rp) - 1, dtype=np.int32), np.diff(rp))
    monkeypatch.setenv("MERCURY_WAIT_POLLS", "0")
    with pytest.raises(McError, match="error flag"):
        dgraph_from_edges(src, col, len(rp) - 1)
    monkeypatch.delenv("MERCURY_WAIT_POLLS")
    with dgraph_from_edges(src, col, len(rp) - 1) as d:
        brp, bcol = d.export_csr()
    assert np.array_equal(brp, rp) and np.array_equal(bcol, col)
