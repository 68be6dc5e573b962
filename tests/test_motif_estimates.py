"""Whole pattern counts of graphs with cliques: the default route, which may stop the
motif sums on the way, against the formulas and the sums taken to their end."""
import numpy as np
import pytest

from brute import random_graph
from conftest import csr_from_edges
from mercury_b200 import DeviceGraph, Graph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def blocks(count, n, p, others=0):
    """`count` random graphs of n vertices side by side, then a path of others."""
    parts = [np.asarray(random_graph(n, p, i), dtype=np.int64).reshape(-1, 2) + i * n
             for i in range(count)]
    a = count * n + np.arange(max(others - 1, 0))
    return csr_from_edges(count * n + others,
                          np.concatenate(parts + [np.stack([a, a + 1], 1)]))


def beside(first, second):
    n = len(first[0]) - 1
    return (np.concatenate([first[0], second[0][1:] + first[0][-1]]),
            np.concatenate([first[1], second[1] + n]).astype(np.int32))


def hubs(n):
    g = Graph.chung_lu(n, 2.1, 8.0, 900.0, seed=n)
    return np.array(g.rowptr), np.array(g.col)


CASES = {
    "cliques": lambda: blocks(20, 60, 1.0),                       # the samples
    "dense blocks": lambda: blocks(10, 90, 0.8),                  # near their line
    "half-filled blocks": lambda: blocks(10, 90, 0.5),            # below it
    "a clique and a path": lambda: blocks(1, 120, 1.0, 3000),     # the estimates
    "a clique and hubs": lambda: beside(blocks(1, 100, 1.0), hubs(4000)),
    "complete": lambda: blocks(1, 100, 1.0),                      # by size
}


@pytest.mark.parametrize("case", CASES)
def test_every_route_gives_the_same_counts(monkeypatch, case):
    rp, col = CASES[case]()
    with DeviceGraph(rp, col) as d:
        got = [d.pattern_count(k) for k in range(1, 9)]
        monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "formula")
        assert got == [d.pattern_count(k) for k in range(1, 9)]
        monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "sparse")
        assert got == [d.pattern_count(k) for k in range(1, 9)]
    if case == "cliques":
        assert got == [orc.pattern(rp, col, k) for k in range(1, 9)] == [0] * 8


def launches(d, patterns):
    out = []
    for k in patterns:
        d.pattern_count(k)
        out.append(d.last_timing.launches)
    return np.array(out)


@pytest.mark.parametrize("case,both", [
    # Complete graphs, too large for the formulas by size (20 of 128 vertices, P1 to
    # P5: 1.3, 47, 24, 1.5 and 47 ms by the sums; 0.4, 1.6, 0.4, 0.4 and 19 by the
    # formulas).
    ("unions", [1, 2, 3, 4, 5]),
    # One of 200 beside a path.
    ("beside a path", [2, 3, 5]),
    ("hubs", []),
])
def test_cliques_send_the_sums_to_the_formulas(monkeypatch, case, both):
    """A count that leaves the sums for the formulas has the launches of both."""
    rp, col = {"unions": lambda: blocks(24, 70, 1.0),
               "beside a path": lambda: blocks(1, 200, 1.0, 5000),
               "hubs": lambda: hubs(20000)}[case]()
    patterns = range(1, 6)
    with DeviceGraph(rp, col) as d:
        got = launches(d, patterns)
        monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "sparse")
        sums = launches(d, patterns)
        monkeypatch.setenv("MERCURY_MOTIF_ROUTE", "formula")
        formulas = launches(d, patterns)
    went = [k for k in patterns if got[k - 1] == sums[k - 1] + formulas[k - 1]]
    stayed = [k for k in patterns if got[k - 1] == sums[k - 1]]
    assert went == both and sorted(went + stayed) == list(patterns)
