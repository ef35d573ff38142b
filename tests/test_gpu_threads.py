"""Engines created, run through captured graphs and destroyed by two host
threads at once, over and over: every run gives its own result.  (One thread's
device-wide wait beside the other's capture used to fail the capture or crash
the process within 150 rounds.)"""
import threading

import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_two_threads_create_run_destroy():
    from gpu_cvt_b200 import engine as eng
    m = mg.icosphere(4)
    cases = [mg.sample_sites(m.V, m.F, n, seed=n) for n in (1200, 2500)]

    def run(S0, graph):
        M = eng.Mesh(m.V, m.F)
        e = eng.Engine(eng.params(k=12, mode=1, profile="ref", use_graph=graph), 1, len(S0), eng.grid_cells(M, len(S0), 12))
        g = e.add(M, S0)
        e.run(3)
        e.run(4)
        out = e.sites(g)
        e.close()
        M.close()
        return out

    ref = [run(S, False) for S in cases]
    bad = []

    def worker(i):
        with torch.cuda.device(0):
            for k in range(40):
                try:
                    if not np.array_equal(run(cases[i], True), ref[i]):
                        bad.append((i, k, "differs"))
                except Exception as ex:  # reported below
                    bad.append((i, k, ex))

    th = [threading.Thread(target=worker, args=(i,)) for i in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join(timeout=120)
    assert not bad, bad
