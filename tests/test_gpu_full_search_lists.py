"""Engines without candidate lists keep each site's list as a row, engines with
them entry by entry: the same lists, triangles and sites, through slots used
again and every reader of the lists."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("k,mode,profile,frame", [(8, 1, "ref", "vertex"), (24, 2, "mixed", "pca"), (32, 0, "fp64", "vertex"),
                                                  (20, 1, "mixed", "vertex")])
def test_rows_and_columns(oracle, k, mode, profile, frame):
    from gpu_cvt_b200 import engine as eng
    m = mg.torus(1.0, 0.3, 60, 30, noise_sigma=0.002, seed=1)
    M = eng.Mesh(m.V, m.F)
    S = [mg.sample_sites(m.V, m.F, n, seed=n) for n in (700, 1300, 33)]
    cells = sum(eng.grid_cells(M, len(s), k) for s in S)
    got = []
    for reuse in (False, True):
        e = eng.Engine(eng.params(k=k, mode=mode, profile=profile, frame=frame, knn_reuse=reuse), 3, 2100, cells)
        a, b = e.add(M, S[0]), e.add(M, S[1])
        e.run(3)
        e.remove(a)
        c = e.add(M, S[2])
        e.run(9)
        out = []
        for g in (b, c):
            out += [e.sites(g), *e.state(g).values(), e.faces(g)[0]]
        got.append(out)
        if frame == "vertex":
            r = oracle.lloyd_run(m.V, m.F, S[1], k, mode, 12, profile=oracle.PROFILES[profile])
            assert np.array_equal(e.state(b)["knn"], r["knn"])
        e.close()
    for x, y in zip(*got):
        assert np.array_equal(x, y)
    M.close()
