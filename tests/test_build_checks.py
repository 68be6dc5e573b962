"""Checks of a CSR built from edge pairs, and builds around whole tiles of keys."""
import numpy as np
import pytest

from mercury_b200 import Graph, dgraph_from_edges
from mercury_b200._ffi import Timing

pytestmark = pytest.mark.gpu


def test_validation_runs_when_asked_for():
    """validate_symmetry checks the built CSR (offsets, entries): two launches
    more than the build alone."""
    g = Graph.rmat(10, 8, seed=2)
    src = np.repeat(np.arange(g.n, dtype=np.int32), np.diff(g.rowptr))
    plain, checked = Timing(), Timing()
    for timing, flag in ((plain, False), (checked, True)):
        with dgraph_from_edges(src, np.array(g.col), g.n, validate_symmetry=flag,
                               timing=timing) as d:
            assert (d.nnz, d.max_degree) == (g.nnz, g.max_degree)
    assert checked.launches == plain.launches + 2


@pytest.mark.parametrize("n", [128, 256, 2048, 4096])  # digits of 8, 9, 8 and 9 bits
@pytest.mark.parametrize("m", [1, 2047, 2048, 2049, 4097])  # around whole tiles of keys
def test_built_csr_at_tile_edges(n, m):
    rng = np.random.default_rng(n + m)
    src, dst = rng.integers(0, n, (2, m)).astype(np.int32)
    keep = src != dst
    key = np.unique(np.concatenate([src[keep].astype(np.int64) * n + dst[keep],
                                    dst[keep].astype(np.int64) * n + src[keep]]))
    with dgraph_from_edges(src, dst, n, validate_symmetry=True) as d:
        rp, col = d.export_csr()
    assert np.array_equal(rp, np.searchsorted(key, np.arange(n + 1, dtype=np.int64) * n))
    assert np.array_equal(col, key % n)
