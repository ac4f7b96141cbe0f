"""GAPBS_PR_PLAIN_LAUNCH=1 (the mode profilers use) launches the kernels of a
sweep loop one by one from the host instead of as a conditional graph.  The
solves that have such a loop -- slice-blocked, batched, and gather solves and
adjoints of large graphs without hubs -- give the same bits either way.  (The
variable is read once per process.)
"""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT, gpu_available

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import hashlib, json, sys
import numpy as np
sys.path[:0] = [%r, %r]
from gapbs_b200 import PageRankEngine
from gapbs_b200.graph import Graph, make_graph
from helpers import seed_teleports
eng = PageRankEngine(0)
out = {}
def note(name, *arrays):
    h = hashlib.sha256()
    for a in arrays:
        h.update(np.ascontiguousarray(a).tobytes())
    out[name] = [h.hexdigest(), eng.last_timing()[2]]
def solve(name, t=None):
    r = eng.run(20, 1e-4, teleport=t)
    note(name, r.scores, r.sweeps, r.err_trace)
g = make_graph("-g 14")
T = seed_teleports(g, 12, np.random.default_rng(2))
eng.set_sweep_layout("blocked", 128, 4096)
eng.upload(g)
solve("blocked")
solve("blocked ppr", T[:, 0].copy())
eng.set_batch_tile(16)
eng.set_batch_schedule(32, 96)
solve("batched", T)
eng.set_sweep_layout("gather")
rng = np.random.default_rng(3)
u, v = rng.integers(0, (1 << 23) + 5, (2, 1 << 24), dtype=np.int32)
eng.upload(Graph.from_edges(u, v, symmetrize=True))
solve("gather")
w = rng.normal(size=eng.n).astype(np.float32)
s = eng.run(20, 1e-4).scores
note("adjoint", *eng.adjoint(w, s, max_iters=5, epsilon=0.0)[:2])
print(json.dumps(out))
""" % (ROOT, os.path.dirname(os.path.abspath(__file__)))


def test_host_launched_sweeps_match(tmp_path):
    if not gpu_available():
        pytest.skip("no CUDA device")
    script = tmp_path / "solves.py"
    script.write_text(SCRIPT)
    res = []
    for mode in ("0", "1"):
        r = subprocess.run([sys.executable, str(script)], capture_output=True, text=True,
                           timeout=600, env=dict(os.environ, GAPBS_PR_PLAIN_LAUNCH=mode))
        assert r.returncode == 0, r.stderr[-2000:]
        res.append(json.loads(r.stdout.strip().splitlines()[-1]))
    assert res[0] == res[1]
    assert len(res[0]) == 5 and all(launches > 1 for _, launches in res[0].values())
