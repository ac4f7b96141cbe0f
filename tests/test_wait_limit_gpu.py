"""Grid barriers whose wait runs out (pr_gpu_set_wait_limit): the call fails
with PR_GPU_ECUDA, and the next one on the same handle and graph gives what it
gave before -- also when a solve was given up with some segments of a long
row counted.  With small limits some CTAs pass a barrier and go on to the
next phase while others have left; no CTA passes the barrier after that.
"""
import numpy as np
import pytest

from gapbs_b200 import PageRankEngine, _pr_abi
from gapbs_b200.graph import make_graph
from gapbs_b200.pagerank import PageRankError
from conftest import gpu_available
from helpers import depths_from_parents

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    if not gpu_available():
        pytest.skip("no CUDA device")
    eng = PageRankEngine(0)
    yield eng
    eng.close()


@pytest.mark.parametrize("weighted", [False, True])
def test_calls_after_a_wait_ran_out(engine, weighted):
    g = make_graph("-g 16")
    n = g.num_nodes
    rng = np.random.default_rng(6)
    ew = rng.uniform(0.5, 1.5, g.num_edges_directed).astype(np.float32) if weighted else None
    engine.upload(g, edge_w=ew)
    w = rng.normal(size=n).astype(np.float32)
    src = int(np.argmax(np.diff(g.out_offsets)))

    def solve():
        r = engine.run(30, 1e-6)
        return [r.scores.view(np.uint32), r.sweeps, r.err_trace]

    scores = engine.run(30, 1e-6).scores
    calls = [solve,
             lambda: list(engine.adjoint(w, scores, max_iters=30, epsilon=1e-6)),
             lambda: [engine.connected_components()],
             lambda: [depths_from_parents(engine.bfs(src), src)]]
    want = [call() for call in calls]

    def equal(a, b):
        return all(np.array_equal(x, y) for x, y in zip(a, b))

    for polls in (0, 1, 2, 3, 4, 8, 16, 0):
        for call, expect in zip(calls, want):
            engine.set_wait_limit(polls)
            try:
                assert equal(call(), expect), polls
                assert polls > 0  # some CTA is always the first to arrive
            except PageRankError as err:
                assert err.code == _pr_abi.PR_GPU_ECUDA and "wait" in str(err)
            finally:
                engine.set_wait_limit(-1)
            for again, expect_again in zip(calls, want):
                assert equal(again(), expect_again), polls


def test_limit_range(engine):
    with pytest.raises(PageRankError) as err:
        engine.set_wait_limit(1 << 31)
    assert err.value.code == _pr_abi.PR_GPU_EINVAL
