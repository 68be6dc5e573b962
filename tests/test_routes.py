"""The routes of whole counts by size (mercury_b200/csrc/routes.h), compiled for
the CPU (tests/routes.cpp)."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
DAG, BITS, PAIRS = range(3)
FORMULA, DENSE, SPARSE = range(3)


@pytest.fixture(scope="module")
def routes():
    out = os.path.join(HERE, "_build", "libroutes.so")
    src = [os.path.join(HERE, "routes.cpp"),
           os.path.join(HERE, "..", "mercury_b200", "csrc", "routes.h")]
    if not os.path.exists(out) or os.path.getmtime(out) < max(map(os.path.getmtime, src)):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", src[0], "-o", out],
                       check=True)
    lib = C.CDLL(out)

    class Routes:
        @staticmethod
        def triangle(n, nnz):
            return lib.triangle_route(C.c_int64(n), C.c_int64(nnz))

        @staticmethod
        def pattern(n, nnz, max_degree, k):
            return lib.pattern_route(C.c_int64(n), C.c_int64(nnz), C.c_int64(max_degree), k)

        @staticmethod
        def samples(n, nnz, max_degree, k):
            return lib.samples(C.c_int64(n), C.c_int64(nnz), C.c_int64(max_degree), k)

        @staticmethod
        def batch_bits(degrees, k):
            n, nnz = len(degrees), sum(degrees)
            return bool(lib.batch_bits(C.c_int64(n), C.c_int64(nnz), C.c_int64(max(degrees)),
                                       C.c_int64(sum(d * d for d in degrees)), k))

    return Routes


@pytest.mark.parametrize("n", [2**30 + 1, 2**31 - 32768, 2**31 - 2])
def test_vertices_beyond_32_bit_loops_keep_the_64_bit_routes(routes, n):
    """The largest graphs a handle takes have more vertices than a 32-bit
    grid-stride loop can step past."""
    assert routes.triangle(n, 1000) == DAG
    assert all(routes.pattern(n, 1000, 40, k) == FORMULA for k in range(1, 9))


def test_at_the_largest_size_of_the_32_bit_loops(routes):
    assert routes.triangle(2**30, 1000) == PAIRS
    assert routes.pattern(2**30, 1000, 40, 1) == SPARSE
    assert routes.pattern(2**30, 2**30 + 1, 40, 1) == FORMULA
    assert routes.pattern(1000, 90000, 46341, 1) == FORMULA


@pytest.mark.parametrize("nnz", [2**31 + 5, 2**32 + 5])
def test_entry_counts_beyond_32_bits_are_no_bit_rows(routes, nnz):
    """Unchecked host arrays may claim any number of entries; the bit rows hold
    row offsets in 32 bits, where such a number would pass for a small one."""
    assert routes.triangle(1000, nnz) == DAG


def complete(n):
    return n, n * (n - 1)


def test_triangles_of_dense_graphs_keep_the_dag(routes):
    """Pairs of up neighbours and bit rows both lose to the DAG where most
    vertices see most others, whatever the number of entries."""
    for n in (400, 512, 600, 1000, 1024):
        assert routes.triangle(*complete(n)) == DAG
    for n, nnz in [(600, 180000), (600, 179886), (1000, 499968), (1000, 500000), (700, 172052)]:
        assert routes.triangle(n, nnz) == DAG
    assert [routes.triangle(*complete(n)) for n in (32, 64, 100, 300)] == [BITS, BITS, PAIRS, PAIRS]
    # Sparse ones, hubs or not, keep the pairs.
    for n, nnz in [(1024, 12014), (8192, 204044), (2048, 177992), (100000, 499200), (2064, 256000)]:
        assert routes.triangle(n, nnz) == PAIRS


def test_batch_jobs_take_bit_rows_where_they_pay(routes):
    """Pattern jobs of a batch: all vertex pairs of a sparse graph of 1,000 vertices
    cost more than its few entries, unless a hub makes the formulas dear; complete
    graphs leave P2 to P4 nothing to test."""
    takes = lambda degrees: [k for k in range(1, 9) if routes.batch_bits(degrees, k)]
    every = list(range(1, 9))
    assert takes([2] * 1000) == []
    assert takes([3] * 1000) == []
    assert takes([10] * 1000) == [2, 3]
    assert takes([100] * 1000) == every
    assert takes([999] + [1] * 999) == [1, 2, 3, 5, 8]
    assert takes([2] * 100) == takes([25] * 500) == takes([10] * 256) == every
    assert takes([99] * 100) == [1, 5, 6, 7, 8]
    assert takes([15] * 16) == every
    assert takes([50] * 1025) == []


def test_patterns_of_near_complete_graphs_keep_the_formulas(routes):
    def formulas(n, percent):
        nnz = n * (n - 1) * percent // 100
        return [k for k in range(1, 9) if routes.pattern(n, nnz, n - 1, k) == FORMULA]

    assert formulas(100, 100) == [1, 2, 3, 4, 5, 6, 8]
    assert formulas(64, 100) == [2, 3, 4, 5, 6, 8]
    assert formulas(200, 100) == formulas(512, 100)[1:] == [2, 3, 4]
    assert formulas(512, 100) == formulas(1000, 100) == [1, 2, 3, 4]
    assert formulas(400, 80) == [1, 3] and formulas(400, 50) == []


def test_samples_are_for_graphs_that_may_be_unions_of_cliques(routes):
    assert [routes.samples(2560, 325120, 127, k) for k in range(1, 9)] == [78] * 3 + [88] + [0] * 4
    assert routes.samples(200, 39800, 199, 1) == 0        # by size
    assert routes.samples(100000, 996680, 200, 1) == 0   # mean 10
    assert routes.samples(60000, 1100000, 17215, 1) == 0  # hubs
