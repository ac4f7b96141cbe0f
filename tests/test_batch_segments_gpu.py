"""Batched sweeps at the lengths that cut a row into segments (128 entries on
small graphs) and at the shortest rows of each lane group, and their first
sweep, which takes rows without a teleport entry as zero: sparse, dense and
all-zero-but-one columns, one sweep, none, and a second solve on the same
work arrays.  Oracle and tolerances of the personalized PageRank tests.
"""
import numpy as np
import pytest

from gapbs_b200 import PageRankEngine
from gapbs_b200.graph import Graph
from conftest import gpu_available
from test_ppr_gpu import check_columns
from test_resident_gpu import hub_graph

pytestmark = pytest.mark.gpu

LENGTHS = (7, 8, 9, 31, 32, 33, 127, 128, 129, 255, 256, 257, 1023, 1025, 4095, 4097)


@pytest.fixture(scope="module")
def engine():
    if not gpu_available():
        pytest.skip("no CUDA device")
    eng = PageRankEngine(0)
    yield eng
    eng.close()


@pytest.mark.parametrize("k", [3, 12, 32, 64])
def test_row_lengths_and_first_sweep(engine, k):
    g = hub_graph(6000, LENGTHS, 5)
    engine.upload(g)
    n = g.num_nodes
    rng = np.random.default_rng(k)
    T = np.zeros((n, k), np.float32)
    T[0, 0] = 1.0                                  # one seed, a hub
    T[:, 1] = rng.random(n).astype(np.float32)     # every row
    T[:, 1] /= T[:, 1].sum()
    for c in range(2, k):
        T[rng.choice(n, 1 + c * 7, replace=False), c] = np.float32(1.0 / (1 + c * 7))
    for iters in (1, 20):
        check_columns(g, T, engine.run(iters, 1e-4, teleport=T), max_iters=iters)
    none = engine.run(0, 1e-4, teleport=T)
    assert np.array_equal(none.scores, T) and not none.sweeps.any()
    sparse = np.ascontiguousarray(T[:, [0] + list(range(2, k))])  # most rows without an entry
    a = engine.run(20, 1e-4, teleport=sparse)
    check_columns(g, sparse, a)
    b = engine.run(20, 1e-4, teleport=sparse)
    assert np.array_equal(a.scores.view(np.uint32), b.scores.view(np.uint32))


@pytest.mark.parametrize("k", [12, 64])
def test_warps_with_segments_only(engine, k):
    """Every row is cut into segments and no warp has ordinary rows between a
    partial and its ticket: the last segment's warp must see all columns of
    the other warps' partials, in every sweep of repeated solves."""
    rng = np.random.default_rng(17)
    n = 400
    u, v = np.divmod(rng.choice(n * n, 120000, replace=False), n)
    g = Graph.from_edges(u.astype(np.int32), v.astype(np.int32))
    assert np.diff(g.in_offsets).min() >= 256
    engine.upload(g)
    T = rng.random((n, k)).astype(np.float32)
    T /= T.sum(axis=0)
    first = engine.run(20, 1e-6, teleport=T)
    check_columns(g, T, first, eps=1e-6)
    for _ in range(20):
        again = engine.run(20, 1e-6, teleport=T)
        assert np.array_equal(first.scores.view(np.uint32), again.scores.view(np.uint32))
        assert np.array_equal(first.err_trace, again.err_trace)
