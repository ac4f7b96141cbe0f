"""GPU adjoint (K4/K5) against the FP64 oracle's adjoint, and through
torch.autograd.

The oracle's adjoint formulas are pinned to central finite differences in
tests/test_adjoint_oracle.py; here the GPU gradients (FP32) must match the
oracle's FP64 gradients computed at the GPU's own forward solution:
  relative L2 error <= 1e-4 for d/dteleport and <= 1e-3 for d/dweights.
"""
import numpy as np
import pytest

import oracle
from gapbs_b200 import PageRankEngine
from gapbs_b200.graph import Graph, make_graph
from conftest import gpu_available
from helpers import in_weights, row_sums, seed_teleports

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    if not gpu_available():
        pytest.skip("no CUDA device")
    eng = PageRankEngine(0)
    yield eng
    eng.close()


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("kind", ["undirected_weighted", "undirected_unit", "directed_weighted"])
def test_adjoint_matches_oracle(engine, kind):
    rng = np.random.default_rng(21)
    if kind.startswith("directed"):
        g = Graph.from_edges(rng.integers(0, 3000, 30000), rng.integers(0, 3000, 30000))
    else:
        g = make_graph("-g 12")
    n, m = g.num_nodes, g.num_edges_directed
    ew = rng.uniform(0.5, 1.5, m).astype(np.float32) if kind.endswith("weighted") else None
    engine.upload(g, edge_w=ew)
    t = seed_teleports(g, 1, rng, max_seeds=200)[:, 0]
    fwd = engine.run(100, 1e-7, teleport=t)
    lw = rng.normal(size=n).astype(np.float32)
    gt, ge, sweeps = engine.adjoint(lw, fwd.scores, max_iters=400, epsilon=1e-7)
    assert 0 < sweeps <= 400
    w64 = None if ew is None else ew.astype(np.float64)
    lam, gt64, gw64, _ = oracle.ppr_adjoint_f64(n, g.out_offsets, g.out_neighbors, lw,
                                                fwd.scores.astype(np.float64), out_w=w64,
                                                max_iters=4000, epsilon=1e-13)
    assert rel_l2(gt, gt64) <= 1e-4
    assert rel_l2(ge, gw64) <= 1e-3


def test_autograd_function(engine):
    torch = pytest.importorskip("torch")
    from gapbs_b200.autograd import PageRankContext, personalized_pagerank
    rng = np.random.default_rng(5)
    g = make_graph("-g 11")
    n, m = g.num_nodes, g.num_edges_directed
    pctx = PageRankContext(g, max_iters=100, epsilon=1e-7, adjoint_max_iters=400,
                           adjoint_epsilon=1e-7)
    t_np = seed_teleports(g, 1, rng)[:, 0]
    t = torch.tensor(t_np, device="cuda", requires_grad=True)
    w = torch.tensor(rng.uniform(0.5, 1.5, m).astype(np.float32), device="cuda", requires_grad=True)
    lw = torch.tensor(rng.normal(size=n).astype(np.float32), device="cuda")
    s = personalized_pagerank(t, w, pctx)
    loss = (lw * s).sum()
    loss.backward()
    assert t.grad.shape == (n,) and w.grad.shape == (m,)
    # FP64 oracle at the same weights
    ew = w.detach().cpu().numpy().astype(np.float64)
    s64, _, _ = oracle.ppr_f64(n, g.in_offsets, g.in_neighbors, g.out_offsets,
                               t_np.astype(np.float64), in_w=in_weights(g, ew),
                               rowsum=row_sums(g, ew), max_iters=2000, epsilon=1e-14)
    assert np.abs(s.detach().cpu().numpy() - s64).sum() <= 1e-5
    _, gt64, gw64, _ = oracle.ppr_adjoint_f64(n, g.out_offsets, g.out_neighbors,
                                              lw.cpu().numpy().astype(np.float64), s64,
                                              out_w=ew, max_iters=4000, epsilon=1e-13)
    assert rel_l2(t.grad.cpu().numpy(), gt64) <= 1e-4
    assert rel_l2(w.grad.cpu().numpy(), gw64) <= 1e-3


def test_set_edge_weights_device(engine):
    """pr_gpu_set_edge_weights_device gives bit for bit what a fresh upload
    of the same weights gives (forward and adjoint); invalid weights are
    refused with PR_GPU_EGRAPH and leave the previous ones; a graph without
    weights refuses the call with PR_GPU_EINVAL."""
    torch = pytest.importorskip("torch")
    from gapbs_b200.pagerank import PageRankError
    rng = np.random.default_rng(8)
    for g in (make_graph("-g 12"),
              Graph.from_edges(rng.integers(0, 3000, 30000), rng.integers(0, 3000, 30000))):
        n, m = g.num_nodes, g.num_edges_directed
        w1 = rng.uniform(0.5, 1.5, m).astype(np.float32)
        w2 = rng.uniform(0.5, 1.5, m).astype(np.float32)
        t = seed_teleports(g, 1, rng)[:, 0]
        lw = rng.normal(size=n).astype(np.float32)
        engine.upload(g, edge_w=w2)
        want = engine.run(100, 1e-7, teleport=t)
        want_gt, want_ge, _ = engine.adjoint(lw, want.scores, max_iters=300, epsilon=1e-7)
        engine.upload(g, edge_w=w1)
        d_w2 = torch.from_numpy(w2).cuda()
        torch.cuda.synchronize()
        engine.set_edge_weights_device(d_w2.data_ptr())
        got = engine.run(100, 1e-7, teleport=t)
        assert np.array_equal(got.scores.view(np.uint32), want.scores.view(np.uint32))
        gt, ge, _ = engine.adjoint(lw, got.scores, max_iters=300, epsilon=1e-7)
        assert np.array_equal(gt, want_gt) and np.array_equal(ge, want_ge)
        bad = d_w2.clone()
        bad[m // 2] = -1.0
        with pytest.raises(PageRankError) as ei:
            engine.set_edge_weights_device(bad.data_ptr())
        assert ei.value.code == -5   # PR_GPU_EGRAPH
        again = engine.run(100, 1e-7, teleport=t)
        assert np.array_equal(again.scores.view(np.uint32), want.scores.view(np.uint32))
    engine.upload(make_graph("-g 10"))
    with pytest.raises(PageRankError) as ei:
        engine.set_edge_weights_device(d_w2.data_ptr())
    assert ei.value.code == -1       # PR_GPU_EINVAL


def test_autograd_training_loop_updates_weights_on_device(engine):
    """Ten SGD steps on the edge weights through torch.autograd: one graph
    upload, then device weight updates only; the final scores match the FP64
    oracle at the final weights."""
    torch = pytest.importorskip("torch")
    from gapbs_b200.autograd import PageRankContext, personalized_pagerank
    rng = np.random.default_rng(13)
    g = make_graph("-g 12")
    n, m = g.num_nodes, g.num_edges_directed
    pctx = PageRankContext(g, max_iters=100, epsilon=1e-7, adjoint_max_iters=300,
                           adjoint_epsilon=1e-7)
    t_np = seed_teleports(g, 1, rng)[:, 0]
    t = torch.tensor(t_np, device="cuda")
    w = torch.tensor(rng.uniform(0.5, 1.5, m).astype(np.float32), device="cuda",
                     requires_grad=True)
    lw = torch.tensor(rng.normal(size=n).astype(np.float32), device="cuda")
    for _ in range(10):
        s = personalized_pagerank(t, w, pctx)
        loss = (lw * s).sum()
        w.grad = None
        loss.backward()
        with torch.no_grad():
            w -= 1e3 * w.grad
            w.clamp_(min=0.05)
    assert pctx.uploads == 1 and pctx.weight_updates == 9
    s = personalized_pagerank(t, w, pctx)
    assert pctx.weight_updates == 10
    ew = w.detach().cpu().numpy().astype(np.float64)
    s64, _, _ = oracle.ppr_f64(n, g.in_offsets, g.in_neighbors, g.out_offsets,
                               t_np.astype(np.float64), in_w=in_weights(g, ew),
                               rowsum=row_sums(g, ew), max_iters=2000, epsilon=1e-14)
    assert np.abs(s.detach().cpu().numpy() - s64).sum() <= 1e-5
    pctx.engine.close()


@pytest.mark.parametrize("kind", ["undirected", "directed", "weighted", "large_uniform"])
def test_outputs_in_place_of_inputs(engine, kind):
    """Gradients written over loss_w or scores are those written elsewhere:
    the edge gradients read the scores after the teleport gradient is done."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(23)
    if kind == "directed":
        g = Graph.from_edges(rng.integers(0, 3000, 30000), rng.integers(0, 3000, 30000))
    elif kind == "large_uniform":   # the sweep launches
        u, v = rng.integers(0, (1 << 23) + 5, (2, 1 << 24), dtype=np.int32)
        g = Graph.from_edges(u, v, symmetrize=True)
    else:
        g = make_graph("-g 12")
    n, m = g.num_nodes, g.num_edges_directed
    ew = rng.uniform(0.5, 1.5, m).astype(np.float32) if kind == "weighted" else None
    engine.upload(g, edge_w=ew)
    w = torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()
    s = torch.from_numpy(rng.random(n).astype(np.float32) / n).cuda()

    def grads(w, s, gt, ge):
        torch.cuda.synchronize()
        engine.adjoint_device(5, 0.0, 0.85, w.data_ptr(), s.data_ptr(), gt.data_ptr(),
                              ge.data_ptr())
        return gt, ge

    gt, ge = grads(w, s, torch.empty(n, device="cuda"), torch.empty(m, device="cuda"))
    assert float(ge.abs().max()) > 0
    s1 = s.clone()
    a, b = grads(w, s1, s1, torch.empty(m, device="cuda"))       # teleport over scores
    assert torch.equal(a, gt) and torch.equal(b, ge)
    w1 = w.clone()
    a, b = grads(w1, s, w1, torch.empty(m, device="cuda"))       # teleport over loss_w
    assert torch.equal(a, gt) and torch.equal(b, ge)
    for first in (0, m - n):                                     # edges over scores
        buf = torch.empty(m, device="cuda")
        buf[first:first + n] = s
        a, b = grads(w, buf[first:first + n], torch.empty(n, device="cuda"), buf)
        assert torch.equal(a, gt) and torch.equal(b, ge)
    buf = torch.empty(n + 8, device="cuda")                      # partly over scores
    buf[8:] = s
    a, b = grads(w, buf[8:], buf[:n], torch.empty(m, device="cuda"))
    assert torch.equal(a, gt) and torch.equal(b, ge)


def test_autograd_fresh_weight_tensors():
    """Weights that are a new tensor every step, in memory that the last one
    left, or another view of the same memory: each solve takes its own."""
    torch = pytest.importorskip("torch")
    if not gpu_available():
        pytest.skip("no CUDA device")
    from gapbs_b200.autograd import PageRankContext, personalized_pagerank
    rng = np.random.default_rng(9)
    g = make_graph("-g 11")
    n, m = g.num_nodes, g.num_edges_directed
    kw = dict(max_iters=100, epsilon=1e-7)
    t = torch.from_numpy(seed_teleports(g, 1, rng)[:, 0]).cuda()
    host = [torch.from_numpy(rng.uniform(0.5, 1.5, m).astype(np.float32)) for _ in range(3)]

    def alone(w):
        pctx = PageRankContext(g, **kw)
        return personalized_pagerank(t, w, pctx).clone()

    want = [alone(w.cuda()) for w in host]
    pctx = PageRankContext(g, **kw)
    for w, expect in zip(host, want):
        d = w.cuda()
        assert torch.equal(personalized_pagerank(t, d, pctx), expect)
        del d                                    # its memory is free again
    both = torch.empty(2 * m, device="cuda")     # one address, two strides
    both[0::2], both[m:] = host[0].cuda(), 1.0
    even, front = both[0::2], both[:m]
    assert even.data_ptr() == front.data_ptr()
    for w in (even, front):
        assert torch.equal(personalized_pagerank(t, w, pctx), alone(w.contiguous()))


def test_autograd_backward_uses_its_own_weights():
    """Two forward passes with different weights on one context, then both
    backward passes: each has the gradients that it has alone.  Weights changed
    in place after a pass: its gradients while the engine still holds the old
    ones, an error once it does not."""
    torch = pytest.importorskip("torch")
    if not gpu_available():
        pytest.skip("no CUDA device")
    from gapbs_b200.autograd import PageRankContext, personalized_pagerank
    rng = np.random.default_rng(10)
    g = make_graph("-g 11")
    n, m = g.num_nodes, g.num_edges_directed
    kw = dict(max_iters=100, epsilon=1e-7)
    t = torch.from_numpy(seed_teleports(g, 1, rng)[:, 0]).cuda().requires_grad_()
    lw = torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()
    weights = [torch.from_numpy(rng.uniform(0.5, 1.5, m).astype(np.float32)).cuda()
               .requires_grad_() for _ in range(2)] + [None]

    def loss(w, pctx):
        return (lw * personalized_pagerank(t, w, pctx)).sum()

    def grads(value, w):
        return torch.autograd.grad(value, (t,) if w is None else (t, w))

    def alone(w):
        return grads(loss(w, PageRankContext(g, **kw)), w)

    pctx = PageRankContext(g, **kw)
    want = [alone(w) for w in weights]
    values = [loss(w, pctx) for w in weights]
    for value, w, expect in zip(values, weights, want):
        assert all(torch.equal(a, b) for a, b in zip(grads(value, w), expect))
    a, b = weights[:2]
    value = loss(a, pctx)
    with torch.no_grad():
        a.mul_(2.0)
    assert all(torch.equal(x, y) for x, y in zip(grads(value, a), want[0]))
    value = loss(b, pctx)
    with torch.no_grad():
        b.mul_(2.0)
    loss(a, pctx)
    with pytest.raises(RuntimeError, match="changed in place"):
        grads(value, b)
