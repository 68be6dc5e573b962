"""Scratch shared by the counts of many handles: blocks of other sizes, from
other streams and threads, kept and given back."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from mercury_b200 import DeviceGraph, Graph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 4])
def test_counts_of_interleaved_handles(threads):
    """Handles of several sizes (bit rows, sparse sums, formulas; scratch from
    the smallest block to 80 MB), each on its own stream, counted in turn and
    from several threads: every count stays its graph's own, also after all
    handles are gone and new ones take the blocks again."""
    specs = [(60, 6.0, 20.0), (300, 8.0, 60.0), (1500, 8.0, 90.0), (6000, 6.0, 120.0),
             (20000, 5.0, 60.0)]
    graphs = [Graph.chung_lu(n, 2.1, mean, cap, seed=n) for n, mean, cap in specs]
    arrays = [(np.array(g.rowptr), np.array(g.col)) for g in graphs]
    want = [[orc.tc(rp, col)] + [orc.pattern(rp, col, p) for p in (1, 4, 7, 8)]
            for rp, col in arrays]

    def work(d):
        return [d.tc_count()] + [d.pattern_count(p) for p in (1, 4, 7, 8)]

    for _ in range(2):
        handles = [DeviceGraph(rp, col) for rp, col in arrays for _ in range(threads)]
        try:
            with ThreadPoolExecutor(threads) as pool:
                for _ in range(3):
                    got = list(pool.map(work, handles))
                    assert got == [w for w in want for _ in range(threads)]
        finally:
            for d in handles:
                d.close()


def test_triangle_counts_of_different_table_sizes_in_threads(monkeypatch):
    """The hub kernel's shared-memory limit belongs to the function: a thread
    with small tables must not lower it under another thread's launch."""
    monkeypatch.setenv("MERCURY_TC_ROUTE", "dag")
    graphs = [Graph.rmat(15, 16, seed=3), Graph.rmat(10, 8, seed=4)]
    want = [orc.tc(np.array(g.rowptr), np.array(g.col)) for g in graphs]

    def work(i):
        with DeviceGraph(graphs[i]) as d:
            return [d.tc_count() for _ in range(400)]

    with ThreadPoolExecutor(2) as pool:
        for got, w in zip(pool.map(work, [0, 1]), want):
            assert set(got) == {w}


def test_route_does_not_depend_on_earlier_counts():
    """Scratch that an earlier count gave back to the pool is free memory: with
    room for it twice, but not four times, the same count takes the motif sums
    every time."""
    import torch
    g = Graph.chung_lu(1000000, 2.1, 9.0, 100.0, seed=6)
    with DeviceGraph(g) as d:
        free = torch.cuda.mem_get_info()[0]
        scratch = 4 * 64 * d.nnz + 40 * d.nnz  # lists at the first guess, and the rest
        fill = torch.empty(max(0, free - int(2.4 * scratch)), dtype=torch.uint8, device="cuda")
        try:
            seen = [(d.pattern_count(1), d.last_timing.launches) for _ in range(3)]
        finally:
            del fill
            torch.cuda.empty_cache()
        assert seen == [(d.pattern_count(1), d.last_timing.launches)] * 3


def test_lists_that_do_not_fit_are_counted_first(monkeypatch):
    """Half of the memory holds the lists' true size but not their first guess:
    a counting pass sizes them (two more launches) before any other route."""
    g = Graph.chung_lu(1000000, 2.1, 9.0, 100.0, seed=6)
    with DeviceGraph(g) as d:
        want, launches = d.pattern_count(7), d.last_timing.launches
        monkeypatch.setenv("MERCURY_DEVICE_BYTES", str(2 * 200 * d.nnz))
        assert (d.pattern_count(7), d.last_timing.launches) == (want, launches + 2)
        monkeypatch.setenv("MERCURY_DEVICE_BYTES", str(1 << 20))
        assert d.pattern_count(7) == want
