"""Motif sums on graphs with a hub above degree 4,096, where the walks of all pairs
and the wheels run in slices: trees and friendship graphs with counts in closed
form, and slices of any length against one another."""
from math import comb

import numpy as np
import pytest

from conftest import csr_from_edges
from mercury_b200 import DeviceGraph, Graph
from oracle import oracle as orc


def spider(d):
    """A centre with d legs of two edges."""
    a = np.arange(d)
    rp, col = csr_from_edges(2 * d + 1, np.concatenate([np.stack([0 * a, 1 + a], 1),
                                                        np.stack([1 + a, 1 + d + a], 1)]))
    claws = comb(d, 3)
    return rp, col, [claws, d * comb(d - 1, 2), 4 * comb(d, 4) + 3 * claws, d * (d - 1), 0, 0, 0, 0]


def friends(t):
    """t triangles that share one vertex."""
    a = np.arange(t)
    rp, col = csr_from_edges(2 * t + 1, np.concatenate([
        np.stack([0 * a, 1 + 2 * a], 1), np.stack([0 * a, 2 + 2 * a], 1),
        np.stack([1 + 2 * a, 2 + 2 * a], 1)]))
    claws = 8 * comb(t, 3)
    return rp, col, [claws, 0, 64 * comb(t, 4) + 3 * claws, 0, 0, 4 * t * (t - 1), 0, 0]


@pytest.mark.parametrize("make", [spider, friends])
@pytest.mark.parametrize("size", [3, 5, 9])
def test_closed_forms_are_the_oracle_counts(make, size):
    rp, col, want = make(size)
    assert [orc.pattern(rp, col, k) for k in range(1, 9)] == want


@pytest.mark.gpu
@pytest.mark.parametrize("make,size", [(spider, 4200), (spider, 12000), (friends, 2100),
                                       (friends, 9000)])
def test_closed_forms_on_hubs(make, size):
    rp, col, want = make(size)
    with DeviceGraph(rp, col) as d:
        assert [d.pattern_count(k) % 2**64 for k in range(1, 9)] == [w % 2**64 for w in want]


@pytest.mark.gpu
def test_long_stages_run_in_slices(monkeypatch):
    """P2, P3, P5 and P6 of a graph with hubs: shorter slices are more launches, and
    the same counts."""
    g = Graph.chung_lu(60000, 2.1, 20.0, 50000.0, seed=4)
    assert g.max_degree > 4096
    patterns = (2, 3, 5, 6)
    seen = {}
    with DeviceGraph(g) as d:
        for ms in ("0.02", "250", "100000"):
            monkeypatch.setenv("MERCURY_PATTERN_SLICE_MS", ms)
            seen[ms] = [(d.pattern_count(k), d.last_timing.launches) for k in patterns]
    assert [c for c, _ in seen["0.02"]] == [c for c, _ in seen["250"]] == \
        [c for c, _ in seen["100000"]]
    assert all(short > long for (_, short), (_, long) in zip(seen["0.02"], seen["100000"]))


@pytest.mark.gpu
def test_walks_in_parts_beyond_the_shared_counters():
    """A hub whose ordered walk goes in parts on a graph of more vertices than the
    shared counters hold (102,400): counters per CTA in global memory."""
    n, spokes = 110000, 30000
    rng = np.random.default_rng(5)
    ends = rng.integers(1, spokes + 1, (90000, 2))
    hub = np.stack([np.zeros(spokes, dtype=np.int64), np.arange(1, spokes + 1)], 1)
    tail = np.stack([np.arange(spokes + 1, n - 1), np.arange(spokes + 2, n)], 1)
    rp, col = csr_from_edges(n, np.concatenate([hub, ends[ends[:, 0] != ends[:, 1]], tail]))
    with DeviceGraph(rp, col) as d:
        assert d.pattern_count(4) == orc.pattern_fast(rp, col, 4)
