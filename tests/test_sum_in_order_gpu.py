"""The device PRVerifier's sum of residuals, which is taken in parallel yet
must be the double that the reference's loop gives: residuals of widely
different sizes (so that many are rounded, halfway cases among them), equal
ones, zeros, one huge one, infinities and NaN, around the sizes of its runs
and groups and the size from which the device adds them.

The graph has no edges, so a vertex's residual is |base - score| and every
term is known exactly: the expected error is numpy's sequential sum.
"""
import numpy as np
import pytest

from gapbs_b200 import PageRankEngine
from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    if not gpu_available():
        pytest.skip("no CUDA device")
    eng = PageRankEngine(0)
    yield eng
    eng.close()


def scores(kind, n, rng):
    x = np.exp2(rng.uniform(-60, 0, n)).astype(np.float32)
    if kind == "halves":      # sums end in halves of the last bit again and again
        x = np.exp2(rng.integers(-56, -2, n)).astype(np.float32)
    elif kind == "equal":
        x[:] = 0.1
    elif kind == "growing":   # the sum passes powers of two all the time
        x = np.sort(np.exp2(rng.uniform(-100, 60, n))).astype(np.float32)
    elif kind == "zeros":
        x[: n - 3] = np.float32(0.15000000596046448) / np.float32(n)
    elif kind == "huge":
        x[n // 2] = 3e38
    elif kind == "inf":
        x[n // 3] = np.inf
    elif kind == "nan":
        x[n // 3], x[n // 2] = np.nan, np.inf
    return x


@pytest.mark.parametrize("n", [(1 << 15) - 1, 1 << 15, 8192 * 5 - 1, 8192 * 5, 8192 * 5 + 1,
                               300_007, 8192 * 256 + 257])
@pytest.mark.parametrize("kind", ["wide", "halves", "equal", "growing", "zeros", "huge", "inf",
                                  "nan"])
def test_sum(engine, n, kind):
    engine.upload_csr(n, np.zeros(n + 1, np.int32), np.zeros(0, np.int32))
    s = scores(kind, n, np.random.default_rng(n))
    damping = np.float32(0.85)
    base = (np.float32(1) - damping) / np.float32(n)
    resid = np.abs(base + damping * np.float32(0) - s)
    want = np.cumsum(resid.astype(np.float64))[-1]    # sequential adds
    got = engine.verify(s, float(damping))
    assert np.isnan(got) if np.isnan(want) else got == want
