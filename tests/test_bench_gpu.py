"""bench.py on a small graph: its step time, by events on the launching
stream, is no shorter than the sweeps that the engine times inside it."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT, gpu_available

pytestmark = pytest.mark.gpu


def test_step_time_covers_the_sweeps():
    if not gpu_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--graph", "-g 20",
                        "--steps", "5", "--warmup", "3", "--no-ppr", "--no-adjoint", "--no-cc",
                        "--no-bfs", "--no-cpu-baseline", "--no-noalloc", "--no-verify",
                        "--e2e-upload-steps", "0"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    d = json.loads(r.stdout.strip().splitlines()[-1])
    sweeps_ms = d["roofline"]["avg_sweep_ms"] * d["config"]["sweeps_per_step"]
    assert d["ms_per_step"] >= sweeps_ms > 0
    assert d["value"] == pytest.approx(d["config"]["num_edges_directed"] *
                                       d["config"]["sweeps_per_step"] / d["ms_per_step"] / 1e6,
                                       rel=1e-2)
