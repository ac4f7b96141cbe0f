"""Four handles on four threads, with graphs whose solves take different amounts
of shared memory: every call succeeds and gives what it gives alone."""
import threading

import numpy as np
import pytest

from gapbs_b200 import PageRankEngine
from gapbs_b200.graph import make_graph
from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layouts", [(("gather", 0, 0), ("gather", 0, 0)),
                                     (("blocked", 49152, 12288), ("blocked", 64, 8192))])
def test_solves_beside_each_other(layouts):
    if not gpu_available():
        pytest.skip("no CUDA device")
    engines, want = [], []
    for args, (name, slice_verts, bin_words) in zip(("-u 16 -k 1", "-u 10 -k 1") * 2, layouts * 2):
        eng = PageRankEngine(0)
        eng.set_sweep_layout(name, slice_verts, bin_words)
        eng.upload(make_graph(args))
        engines.append(eng)
        want.append(eng.run(2, 0.0).scores.view(np.uint32))
    failures = []

    def work(i):
        try:
            for _ in range(2000):
                if not np.array_equal(engines[i].run(2, 0.0).scores.view(np.uint32), want[i]):
                    failures.append((i, "scores differ"))
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            failures.append((i, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for eng in engines:
        eng.close()
    assert not failures, failures[:4]
