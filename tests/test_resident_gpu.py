"""The resident gather solve (one launch for init, sweeps and write-back) at
the sizes where its split of the rows can go wrong: around the length that
cuts a row into segments, the shortest rows of each lane group, the number of
contribs held in shared memory, and graphs small enough for one CTA.  Plain
solves against the oracle with the tolerances of the plain parity tests, the
adjoint (whose out-rows of a directed graph are taken in another order) with
those of the adjoint tests.
"""
import numpy as np
import pytest

import oracle
from gapbs_b200 import PageRankEngine
from gapbs_b200.graph import Graph, make_graph
from conftest import gpu_available
from helpers import seed_teleports

pytestmark = pytest.mark.gpu

TILE = 40960


@pytest.fixture(scope="module")
def engine():
    if not gpu_available():
        pytest.skip("no CUDA device")
    eng = PageRankEngine(0)
    eng.set_sweep_layout("gather")
    yield eng
    eng.close()


def check(engine, g, max_iters=20, epsilon=1e-4):
    res = engine.run(max_iters, epsilon)
    s32, k32, _ = oracle.pr_pull_f32(g, max_iters, epsilon)
    s64, _, _ = oracle.pr_pull_f64(g, max_iters, epsilon)
    assert int(res.sweeps[0]) == k32
    assert np.all(np.abs(res.scores - s64) <= 2e-5 * np.abs(s64) + 1e-10)
    ref_l1 = float(np.abs(s32.astype(np.float64) - s64).sum())
    assert float(np.abs(res.scores.astype(np.float64) - s64).sum()) <= 4 * ref_l1 + 1e-7
    again = engine.run(max_iters, epsilon)
    assert np.array_equal(res.scores.view(np.uint32), again.scores.view(np.uint32))
    assert np.array_equal(res.err_trace, again.err_trace)
    return res


def hub_graph(n, lengths, seed):
    """Directed: row and out-row i of the first len(lengths) vertices have
    lengths[i] different neighbours each; a sparse rest."""
    rng = np.random.default_rng(seed)
    u, v = [rng.integers(0, n, 2 * n)], [rng.integers(0, n, 2 * n)]
    k = len(lengths)
    keep = (u[0] >= k) & (v[0] >= k)
    u[0], v[0] = u[0][keep], v[0][keep]
    for i, length in enumerate(lengths):
        for a, b in ((u, v), (v, u)):
            a.append(np.full(length, i))
            b.append(k + rng.choice(n - k, length, replace=False))
    return Graph.from_edges(np.concatenate(u).astype(np.int32),
                            np.concatenate(v).astype(np.int32))


@pytest.mark.parametrize("lengths", [(1023, 1024, 1025, 2047, 2048, 2049),
                                     (7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129)])
def test_row_classes(engine, lengths):
    g = hub_graph(5000, lengths, 3)
    engine.upload(g)
    check(engine, g)
    rng = np.random.default_rng(4)
    t = seed_teleports(g, 1, rng)[:, 0]
    fwd = engine.run(100, 1e-7, teleport=t)
    w = rng.normal(size=g.num_nodes).astype(np.float32)
    gt, ge, sweeps = engine.adjoint(w, fwd.scores, max_iters=400, epsilon=1e-7)
    assert 0 < sweeps <= 400
    _, gt64, gw64, _ = oracle.ppr_adjoint_f64(g.num_nodes, g.out_offsets, g.out_neighbors, w,
                                              fwd.scores.astype(np.float64), max_iters=4000,
                                              epsilon=1e-13)
    assert np.linalg.norm(gt - gt64) <= 1e-4 * np.linalg.norm(gt64)
    assert np.linalg.norm(ge - gw64) <= 1e-3 * np.linalg.norm(gw64)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 33, TILE - 1, TILE, TILE + 1, TILE + 3])
def test_tile_edges(engine, n):
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, (2, 6 * n)).astype(np.int32)
    u[:1], v[:1] = 0, n - 1
    g = Graph.from_edges(u, v)
    engine.upload(g)
    check(engine, g)
    r = engine.run(0, 1e-4)
    assert int(r.sweeps[0]) == 0 and np.all(r.scores == np.float32(1) / np.float32(g.num_nodes))


@pytest.mark.parametrize("args", ["-g 15", "-g 17", "-u 19"])
def test_row_class_sets(engine, args):
    """Graphs of each of the three sets of row classes (32, 750 and 3,500
    entries a warp of a full grid)."""
    g = make_graph(args)
    engine.upload(g)
    check(engine, g)


def test_long_trace(engine):
    """More sweeps than the page-locked trace holds."""
    g = make_graph("-g 10")
    engine.upload(g)
    r = engine.run(5000, 0.0)
    assert int(r.sweeps[0]) == 5000 and r.err_trace.shape == (5000, 1)
    short = engine.run(50, 0.0)
    assert np.array_equal(r.err_trace[:50], short.err_trace)


def test_large_uniform_graph_keeps_sweep_launches(engine):
    """Over 2^23 vertices without hubs: the sweep kernels in a loop graph, plain
    and adjoint, at a fixed number of sweeps."""
    n = (1 << 23) + 5
    rng = np.random.default_rng(8)
    u, v = rng.integers(0, n, (2, 2 * n), dtype=np.int32)
    u[0] = n - 1
    g = Graph.from_edges(u, v, symmetrize=True)
    engine.upload(g)
    res = engine.run(4, 0.0)
    s64, _, _ = oracle.pr_pull_f64(g, 4, 0.0)
    assert int(res.sweeps[0]) == 4
    assert np.all(np.abs(res.scores - s64) <= 2e-5 * np.abs(s64) + 1e-10)
    w = rng.normal(size=g.num_nodes).astype(np.float32)
    gt, ge, sweeps = engine.adjoint(w, res.scores, max_iters=5, epsilon=0.0)
    assert sweeps == 5
    _, gt64, gw64, _ = oracle.ppr_adjoint_f64(g.num_nodes, g.out_offsets, g.out_neighbors, w,
                                              res.scores.astype(np.float64), max_iters=5,
                                              epsilon=0.0)
    assert np.linalg.norm(gt - gt64) <= 1e-4 * np.linalg.norm(gt64)
    assert np.linalg.norm(ge - gw64) <= 1e-3 * np.linalg.norm(gw64)


def test_many_vertices_few_edges(engine):
    """Init, sweeps and write-back of a graph with hardly any edges use the
    whole GPU: 16 M vertices pass through DRAM a few times, well under a
    millisecond (several with a CTA per 1,024 entries, a few SMs only)."""
    n = 1 << 24
    rng = np.random.default_rng(10)
    u, v = rng.integers(0, n, (2, 3000), dtype=np.int32)
    u[0] = n - 1
    g = Graph.from_edges(u, v, symmetrize=True)
    engine.upload(g)
    check(engine, g)
    ms = []
    for _ in range(5):
        engine.run(20, 1e-4)
        ms.append(engine.last_timing()[1])
    print("device ms a solve:", ms)
    assert min(ms) < 1.5


def test_kernel_times_are_of_the_solve_that_runs(engine):
    """pr_gpu_sweep_kernel_times on the gather layout times the one launch that
    ordinary solves are."""
    engine.upload(make_graph("-g 16"))
    res = engine.run(20, 1e-4)
    assert engine.last_timing()[2] == 1
    ms, sweeps = engine.sweep_kernel_times(20, 1e-4)
    sweep_ms, total_ms, launches = engine.last_timing()
    assert launches == 1 and len(ms) == 1 and sweeps == int(res.sweeps[0])
    assert 0 < ms[0] * sweeps <= total_ms and ms[0] * sweeps == pytest.approx(sweep_ms)
