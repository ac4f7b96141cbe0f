"""Workloads whose time is measured, through the package's public entry points.

Each case is one call (or one training step) that a user's program makes on a
graph it keeps on the GPU.  Graphs are made from the seed: R-MAT with the
suite's quadrant probabilities (0.57 / 0.19 / 0.19, as pr_spmv -g) or
uniform (as -u), with randomly relabelled ids, symmetrised and squished like
the reference's builder does; `directed` keeps one direction per edge, as a
web or citation graph has.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the graph on the engine, and the call's buffers
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   what run returns, in 64 bits with plain torch
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from gapbs_b200 import Graph, PageRankEngine
from gapbs_b200.autograd import PageRankContext, personalized_pagerank

DEV = "cuda:0"
DAMPING = float(np.float32(0.85))
EPSILON, MAX_ITERS = 1e-4, 20                  # pr_spmv's defaults
TRAIN = dict(max_iters=100, epsilon=1e-7, adjoint_max_iters=300, adjoint_epsilon=1e-7)
LEARNING_RATE = 1e-3
CHUNK = 1 << 26                                # edges generated at a time


def _case(name, kind, n, degree, uniform=False, directed=False, cols=1, host=False):
    return {"name": name, "kind": kind, "n": n, "degree": degree, "uniform": uniform,
            "directed": directed, "cols": cols, "host": host}


def listed():
    return [
        # PageRank on a graph of a thousand vertices (pr_spmv -g 10, the
        # suite's own test): latency and launches are all there is
        _case("pagerank_2p10", "pagerank", 1 << 10, 16),
        # pr_spmv -g 16: a community or product graph that fits the caches
        _case("pagerank_2p16", "pagerank", 1 << 16, 16),
        # the call a reference user makes: scores back in host memory; an
        # odd vertex count and edge factor
        _case("pagerank_host_3m", "pagerank", 3_000_017, 13, host=True),
        # pr_spmv -u 24: no hubs, no locality
        _case("pagerank_uniform_2p24", "pagerank", 1 << 24, 16, uniform=True),
        # pr_spmv -g 25, the headline graph (1.05e9 directed edges)
        _case("pagerank_2p25", "pagerank", 1 << 25, 16),
        # 64 personalized vectors at once on a directed-edge count of 1.3e8:
        # the offline job of a recommender
        _case("ppr_64_2p22", "ppr", 1 << 22, 16, cols=64),
        # a small batch of queries on a directed graph of odd size
        _case("ppr_12_directed_300k", "ppr", 300_007, 11, directed=True, cols=12),
        # a step of training edge weights: forward, adjoint, update
        _case("train_2p20", "train", 1 << 20, 16),
        # the same on a small directed graph
        _case("train_directed_50k", "train", 50_021, 9, directed=True),
        # connected components and breadth-first search of a social graph
        _case("components_2p23", "components", 1 << 23, 16),
        _case("bfs_2p23", "bfs", 1 << 23, 16),
        # the check behind -v: PRVerifier's error of given scores
        _case("verify_2p22", "verify", 1 << 22, 16),
    ]


# kind -> (smallest n, largest n, most n * degree, share of draws)
_RANGES = {
    "pagerank": (1_000, 1 << 25, 1 << 29, 5),
    "ppr": (1_000, 1 << 22, 1 << 26, 2),
    "train": (1_000, 1 << 20, 1 << 24, 2),
    "components": (1_000, 1 << 23, 1 << 27, 1),
    "bfs": (1_000, 1 << 23, 1 << 27, 1),
    "verify": (1_000, 1 << 22, 1 << 26, 1),
}


def draw(rng):
    kind = rng.choice([k for k, r in _RANGES.items() for _ in range(r[3])])
    lo, hi, most, _ = _RANGES[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    degree = min(rng.randint(4, 16 if kind == "train" else 28), most // n)
    plain = kind in ("pagerank", "train")
    uniform = plain and rng.random() < 0.25
    if uniform:
        n = min(n, 1 << 24)
    directed = kind in ("pagerank", "ppr", "train") and rng.random() < 0.3
    cols = int(round(math.exp(rng.uniform(0, math.log(64))))) if kind == "ppr" else 1
    c = _case("", kind, n, degree, uniform, directed, cols,
              kind == "pagerank" and rng.random() < 0.3)
    del c["name"]
    return c


# -- inputs ---------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _edges(case, gen):
    """Source and target of n * degree random edges (int32)."""
    n, m = case["n"], case["n"] * case["degree"]
    if case["uniform"]:
        return tuple(torch.randint(0, n, (m,), device=DEV, dtype=torch.int32, generator=gen)
                     for _ in range(2))
    levels = max(1, (n - 1).bit_length())
    relabel = (torch.randperm(1 << levels, device=DEV, generator=gen) % n).int()
    ends = [[], []]
    for at in range(0, m, CHUNK):
        k = min(CHUNK, m - at)
        u = torch.zeros(k, device=DEV, dtype=torch.int32)
        v = torch.zeros(k, device=DEV, dtype=torch.int32)
        for _ in range(levels):
            r = torch.rand(k, device=DEV, generator=gen)
            lower = r >= 0.76
            u.mul_(2).add_(lower)
            v.mul_(2).add_(((r >= 0.57) & ~lower) | (r >= 0.95))
        ends[0].append(relabel[u])
        ends[1].append(relabel[v])
    return torch.cat(ends[0]), torch.cat(ends[1])


def _csr(u, v, n):
    """Rows u, sorted neighbours v, no duplicates, no self-loops: (offsets, neighbours)."""
    bits = max(1, (n - 1).bit_length())
    key = ((u.long() << bits) | v)[u != v]
    key = torch.unique(key)
    rows = torch.arange(n + 1, device=DEV) << bits
    off = torch.searchsorted(key, rows).int()
    return off, (key & ((1 << bits) - 1)).int()


def _graph(case, gen):
    """(n, out-CSR, in-CSR) on the GPU; an undirected graph has one CSR."""
    u, v = _edges(case, gen)
    n = case["n"]
    if case["directed"]:
        return n, _csr(u, v, n), _csr(v, u, n)
    out = _csr(torch.cat([u, v]), torch.cat([v, u]), n)
    return n, out, out


def _host(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    return h.copy_(t)


def _engine(n, out, inc):
    eng = PageRankEngine(0)
    host = [_host(x).numpy() for x in out]
    host += [_host(x).numpy() for x in inc] if inc is not out else [None, None]
    eng.upload_csr(n, *host)
    return eng


def _teleports(case, gen):
    """One column per vector: 1 .. 4096 seed vertices (log-uniform) of equal weight."""
    n, k = case["n"], case["cols"]
    most = math.log2(min(4096, max(2, n // 8)))
    sizes = torch.exp2(torch.rand(k, device=DEV, generator=gen) * most).round().long()
    t = torch.zeros(n, k, device=DEV)
    for c, size in enumerate(sizes.tolist()):
        t[torch.randperm(n, device=DEV, generator=gen)[:size], c] = 1.0 / size
    return t if k > 1 else t[:, 0].contiguous()


def _train_inputs(case, seed):
    """Edge list of exactly n * degree different edges (so that gradients have
    one size whatever the seed), and the tensors of a step."""
    gen = _generator(seed)
    n, m = case["n"], case["n"] * case["degree"]
    bits = max(1, (n - 1).bit_length())
    last = ((n - 2) << bits) | (n - 1)           # always there: the largest id is n - 1
    key = torch.empty(0, device=DEV, dtype=torch.int64)
    while key.numel() < m:
        u, v = _edges(case, gen)
        if not case["directed"]:
            u, v = torch.minimum(u, v), torch.maximum(u, v)
        new = ((u.long() << bits) | v)[u != v]
        key = torch.unique(torch.cat([key, new[new != last]]))
    key = key[torch.randperm(key.numel(), device=DEV, generator=gen)[:m]]
    key[0] = last
    u, v = (key >> bits).int(), (key & ((1 << bits) - 1)).int()
    t = torch.rand(n, device=DEV, generator=gen)
    w = torch.rand(m if case["directed"] else 2 * m, device=DEV, generator=gen) + 0.5
    loss = torch.randn(n, device=DEV, generator=gen)
    return u, v, t / t.sum(), w, loss


def prepare(case, seed):
    s = SimpleNamespace(kind=case["kind"], cols=case["cols"], host=case["host"])
    if s.kind == "train":
        u, v, t, w, s.loss = _train_inputs(case, seed)
        g = Graph.from_edges(u.cpu().numpy(), v.cpu().numpy(), symmetrize=not case["directed"])
        s.teleport, s.weights = t.requires_grad_(), w.requires_grad_()
        s.context = PageRankContext(g, **TRAIN)
        s.context.ensure_weights(s.weights)
        return s
    gen = _generator(seed)
    n, out, inc = _graph(case, gen)
    s.engine = _engine(n, out, inc)
    if s.kind == "ppr":
        s.teleport = _teleports(case, gen)
        s.scores = torch.empty_like(s.teleport)
    elif s.kind == "pagerank":
        s.scores = (torch.empty(n, pin_memory=True).numpy() if s.host
                    else torch.empty(n, device=DEV))
    elif s.kind == "verify":
        p, _ = _transition(n, out, inc)
        s.given = _solve(p, torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64),
                         MAX_ITERS, EPSILON)[0].float().cpu().numpy()
    else:
        s.result = torch.empty(n, device=DEV, dtype=torch.int32)
        nbr = out[1]
        s.source = int(nbr[torch.randint(nbr.numel(), (1,), device=DEV, generator=gen)])
    return s


def run(s):
    if s.kind == "train":
        scores = personalized_pagerank(s.teleport, s.weights, s.context)
        gt, gw = torch.autograd.grad((scores * s.loss).sum(), (s.teleport, s.weights))
        with torch.no_grad():
            s.weights.sub_(gw, alpha=LEARNING_RATE)
        return {"scores": scores.detach(), "grad_teleport": gt, "grad_weights": gw}
    if s.kind == "pagerank" and s.host:
        r = s.engine.run(MAX_ITERS, EPSILON, out=s.scores)
        return {"scores": r.scores, "sweeps": r.sweeps}
    if s.kind == "pagerank":
        sweeps, _ = s.engine.run_device(MAX_ITERS, EPSILON, DAMPING, 1, None,
                                        s.scores.data_ptr())
        return {"scores": s.scores, "sweeps": sweeps}
    if s.kind == "ppr":
        sweeps, _ = s.engine.run_device(MAX_ITERS, EPSILON, DAMPING, s.cols,
                                        s.teleport.data_ptr(), s.scores.data_ptr())
        return {"scores": s.scores, "sweeps": sweeps}
    if s.kind == "components":
        s.engine.connected_components_device(s.result.data_ptr())
        return {"labels": s.result}
    if s.kind == "bfs":
        # which of several parents of equal depth is taken is a race, here as
        # in the reference; what a search reaches, and in how many steps, is not
        steps = s.engine.bfs_device(s.source, s.result.data_ptr())
        return {"reached": s.result >= 0, "steps": steps}
    return {"error": s.engine.verify(s.given)}


# -- what a pass cannot do without ------------------------------------------------

def work(case):
    """Sweeps are those the suite's graphs take to the given epsilon; a sweep
    reads every neighbour id, offset, degree, old score and contribution once
    and writes scores and contributions once.  Duplicate edges (2 to 40 % of
    the drawn ones, more on small graphs) are taken off roughly."""
    n, k = case["n"], case["cols"]
    kept = 1.0 if case["uniform"] else min(0.97, 0.4 + 0.023 * math.log2(n))
    m = n * case["degree"] * kept * (1 if case["directed"] else 2)
    kind = case["kind"]
    if kind == "pagerank":
        sweeps = 6 if case["uniform"] else 8
        return {"bytes": sweeps * (4 * m + 20 * n) + 12 * n, "flops": sweeps * (m + 5 * n)}
    if kind == "ppr":
        sweeps = 12
        return {"bytes": sweeps * (4 * m + 4 * n + 12 * n * k) + 8 * n * k,
                "flops": sweeps * k * (m + 5 * n)}
    if kind == "train":
        sweeps, m = 130, n * case["degree"] * (1 if case["directed"] else 2)
        return {"bytes": sweeps * (8 * m + 24 * n) + 20 * m, "flops": sweeps * (2 * m + 6 * n)}
    if kind == "verify":
        return {"bytes": 4 * m + 16 * n, "flops": m + 4 * n}
    # Afforest and the direction-optimizing search look at a few neighbours a vertex
    return {"bytes": 20 * n, "flops": 2 * n}


# -- the same in 64 bits, with plain torch ----------------------------------------

def _matrix(off, nbr, values, n):
    return torch.sparse_csr_tensor(off, nbr, values, size=(n, n), check_invariants=False)


def _transition(n, out, inc):
    """P^T with P[v, u] = 1 / out_degree(v), and the in-CSR it is built on."""
    degree = (out[0][1:] - out[0][:-1]).double()
    return _matrix(inc[0], inc[1], (1.0 / degree)[inc[1]], n), degree


def _solve(p, t, max_iters, epsilon, norm=1.0, scale=1.0 - DAMPING):
    """x = scale t + d P x from x = t; a column stops when its L1 change < epsilon."""
    x, base = t, t * scale
    live = torch.ones(t.shape[1:], device=t.device, dtype=torch.bool)
    sweeps = torch.zeros(t.shape[1:], device=t.device, dtype=torch.int32)
    for _ in range(max_iters):
        new = base + DAMPING * (p @ x)
        change = (new - x).abs().sum(0)
        x = torch.where(live, new, x)
        sweeps += live
        live = live & (change >= epsilon * norm)
        if not bool(live.any()):
            break
    return x, sweeps


def _exact_train(case, seed):
    n = case["n"]
    u, v, *tensors = _train_inputs(case, seed)
    if not case["directed"]:
        u, v = torch.cat([u, v]), torch.cat([v, u])
    off, nbr = _csr(u, v, n)
    t, w, loss = (x.double() for x in tensors)
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (off[1:] - off[:-1]).long())
    total = torch.zeros(n, device=DEV, dtype=torch.float64).index_add_(0, rows, w)
    p = _matrix(off, nbr, w / total[rows], n)
    order = torch.argsort((nbr.long() << 32) | rows)
    pt = _matrix(torch.searchsorted(nbr[order].contiguous(),
                                    torch.arange(n + 1, device=DEV, dtype=torch.int32)).int(),
                 rows[order].int(), (w / total[rows])[order], n)
    s, _ = _solve(pt, t, TRAIN["max_iters"], TRAIN["epsilon"])
    lam, _ = _solve(p, loss, TRAIN["adjoint_max_iters"], TRAIN["adjoint_epsilon"],
                    float(loss.abs().sum()), 1.0)
    gw = DAMPING * (s / total)[rows] * (lam[nbr] - (p @ lam)[rows])
    return {"scores": s, "grad_teleport": (1.0 - DAMPING) * lam, "grad_weights": gw}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] not in ("pagerank", "ppr"):
        return None      # labels, reached vertices, a verdict: nothing to round
    gen = _generator(seed)
    n, out, inc = _graph(case, gen)
    p, _ = _transition(n, out, inc)
    t = (_teleports(case, gen).double() if case["kind"] == "ppr"
         else torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64))
    x, _ = _solve(p, t, MAX_ITERS, EPSILON)
    return {"scores": x, "sweeps": None}
