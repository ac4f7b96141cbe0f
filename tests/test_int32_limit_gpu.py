"""Graphs of 2^31 - 9 entries, the most an upload takes: every loop over a
row's entries that steps past the end of the last rows passes 2^31.

Row u lists vertex u ^ 1 all over, so one step of any solve is one product per
vertex and the expected values follow in FP64 without the graph.  Rows of
8,192 entries are cut into segments by the solves and take a block each in the
verifier; rows of 2,048 take one warp there, and the last (2,039 entries) one
warp of the resident solve.

Tolerances: a float sum of 8,192 equal terms in a tree of 4-entry chunks is
within 70 roundings of the exact one (5 sweeps: 5 x 70 x 6e-8 = 2e-5);
sequential float adds of the verifier are within 8,192 roundings (5e-4).
"""
import os

import numpy as np
import pytest

from gapbs_b200 import PageRankEngine
from conftest import gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.fullsize]

M = (1 << 31) - 9
D = float(np.float32(0.85))


@pytest.fixture(scope="module", params=[8192, 2048])
def loaded(request):
    if not gpu_available():
        pytest.skip("no CUDA device")
    if os.sysconf("SC_PAGE_SIZE") * os.sysconf("SC_PHYS_PAGES") < (48 << 30):
        pytest.skip("needs 48 GB of host memory")
    deg = request.param
    n = (1 << 31) // deg
    lens = np.full(n, deg, np.int64)
    lens[-1] -= 9
    off = np.zeros(n + 1, np.int32)
    off[1:] = np.cumsum(lens)
    assert off[-1] == M
    mate = np.arange(n, dtype=np.int32) ^ 1
    eng = PageRankEngine(0)
    eng.set_sweep_layout("gather")
    eng.upload_csr(n, off, np.repeat(mate, lens))
    yield eng, lens.astype(np.float64), mate
    eng.close()


def expected(t, lens, mate, sweeps):
    s = t.astype(np.float64)
    for _ in range(sweeps):
        s = (1 - D) * t + D * (lens / lens[mate])[:, None] * s[mate]
    return s


@pytest.mark.parametrize("cols", [1, 8])
def test_solves(loaded, cols):
    eng, lens, mate = loaded
    eng.set_batch_tile(8)
    t = np.random.default_rng(cols).random((lens.size, cols)).astype(np.float32)
    res = eng.run(5, 0.0, teleport=t[:, 0].copy() if cols == 1 else t)
    want = expected(t, lens, mate, 5)
    np.testing.assert_allclose(res.scores.reshape(lens.size, cols), want, rtol=2e-5)


def test_adjoint(loaded):
    torch = pytest.importorskip("torch")
    eng, lens, mate = loaded
    n = lens.size
    rng = np.random.default_rng(3)
    w, s = rng.random((2, n)).astype(np.float32)
    d_w, d_s = torch.from_numpy(w).cuda(), torch.from_numpy(s).cuda()
    gt = torch.empty(n, device="cuda")
    ge = torch.full((M,), 7.0, device="cuda")
    torch.cuda.synchronize()
    eng.adjoint_device(5, 0.0, D, d_w.data_ptr(), d_s.data_ptr(), gt.data_ptr(), ge.data_ptr())
    lam = w.astype(np.float64)
    for _ in range(5):
        lam = w + D * lam[mate]
    np.testing.assert_allclose(gt.cpu().numpy(), (1 - D) * lam, rtol=2e-5)
    # all entries of a row lead to one vertex: lambda there less its mean is 0
    assert float(ge.abs().max()) <= 1e-12
    del ge
    torch.cuda.empty_cache()


def test_verify(loaded):
    eng, lens, mate = loaded
    s = np.random.default_rng(4).random(lens.size).astype(np.float32)
    s64 = s.astype(np.float64)
    want = np.abs((1 - D) / lens.size + D * (lens / lens[mate]) * s64[mate] - s64).sum()
    assert abs(eng.verify(s) - want) <= 5e-4 * s64.sum()


def test_components_and_search(loaded):
    eng, lens, mate = loaded
    n = lens.size
    ids = np.arange(n, dtype=np.int32)
    assert np.array_equal(eng.connected_components(), ids & ~1)
    for src in (0, n - 1):
        parent = eng.bfs(src)
        want = np.full(n, -1, np.int32)
        want[[src, src ^ 1]] = src
        assert np.array_equal(parent, want)
