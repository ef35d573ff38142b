"""Host threads that capture graphs beside threads that create and release
engines, meshes, streams, events, graphs and cached memory: every round ends,
every result is its own."""
import threading

import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ROUNDS = 160


def test_captures_beside_releases():
    from gpu_cvt_b200 import _lib
    from gpu_cvt_b200 import engine as eng
    m = mg.icosphere(4)
    M = eng.Mesh(m.V, m.F)
    sites = {n: mg.sample_sites(m.V, m.F, n, seed=n) for n in (300, 1200, 2500)}

    def prm(graph=True):
        return eng.params(k=12, mode=1, profile="ref", use_graph=graph)

    def alone(n, graph=True, mesh=None):
        e = eng.Engine(prm(graph), 1, n, eng.grid_cells(M, n, 12))
        g = e.add(mesh or M, sites[n])
        e.run(3)
        e.run(4)
        out = e.sites(g)
        e.close()
        return out

    want = {n: alone(n, False) for n in sites}

    def capture(n):
        assert np.array_equal(alone(n), want[n])

    def extents():                           # the covered slots grow and shrink: kept graphs change hands
        e = eng.Engine(prm(), 2, 60000, 240000)
        a = e.add(M, sites[300])
        e.run(7)
        b = e.add(M, sites[2500])
        e.run(7)
        assert np.array_equal(e.sites(a), alone_twice)
        assert np.array_equal(e.sites(b), want[2500])
        e.remove(b)
        e.profile(2)
        e.close()

    def batch():
        out = eng.remesh_batch([m.V] * 3, [m.F] * 3, [sites[n] for n in sites], prm(), 7)
        for o, n in zip(out, sites):
            assert np.array_equal(o, want[n])
        mesh = eng.Mesh(m.V, m.F)
        mesh.close()
        _lib.call("cvt_release_cached_memory")

    e = eng.Engine(prm(False), 1, 300, eng.grid_cells(M, 300, 12))
    g = e.add(M, sites[300])
    e.run(14)
    alone_twice = e.sites(g)
    e.close()

    jobs = [lambda: capture(1200), lambda: capture(2500), extents, batch]
    done, bad = [0] * len(jobs), []

    def worker(i):
        with torch.cuda.device(0):
            for _ in range(ROUNDS):
                try:
                    jobs[i]()
                except Exception as ex:      # reported below
                    bad.append((i, done[i], repr(ex)))
                done[i] += 1

    th = [threading.Thread(target=worker, args=(i,), daemon=True) for i in range(len(jobs))]
    for t in th:
        t.start()
    for t in th:
        t.join(timeout=120)
    assert not any(t.is_alive() for t in th), f"rounds ended: {done}"
    assert not bad, bad[:5]
    assert done == [ROUNDS] * len(jobs)
    M.close()
