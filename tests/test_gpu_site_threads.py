"""Vertex search and projection with one thread per site, which engines that
cover more than 32,768 sites run, on the small cases of the kernels with lanes:
a second segment keeps the covered slots above that line.  Bit for bit against
the oracle, through long rings, ties, deferred searches and freezing."""
import numpy as np
import pytest

import test_gpu_site_order as order
from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CAPACITY = 33000                             # covered while a quarter of it is in use


@pytest.fixture(scope="module")
def eng():
    from gpu_cvt_b200 import engine
    assert torch.cuda.is_available()
    return engine


def _run(eng, m, S0, k, mode, iters, profile, reuse=True, **shapes):
    """The sites' run beside a filler segment, whose slots come first."""
    f = mg.icosphere(3)
    F, M = eng.Mesh(f.V, f.F), eng.Mesh(m.V, m.F)
    n = CAPACITY // 4 + 50
    e = eng.Engine(eng.params(k=k, mode=mode, profile=profile, knn_reuse=reuse, **shapes), 2, CAPACITY,
                   eng.grid_cells(F, n, k) + eng.grid_cells(M, len(S0), k))
    e.add(F, mg.sample_sites(f.V, f.F, n, seed=9))
    g = e.add(M, S0)
    e.run(iters)
    S = e.sites_f64(g) if profile == "fp64" else e.sites(g)
    st = e.state(g)
    e.close()
    F.close()
    M.close()
    return S, st


def _poles(nu=90, nv=24):
    """A sphere of latitudes and longitudes: rings of nu faces at the poles."""
    th, ph = np.pi * np.arange(1, nv) / nv, 2 * np.pi * np.arange(nu) / nu
    P = np.stack([np.outer(np.sin(th), np.cos(ph)), np.outer(np.sin(th), np.sin(ph)), np.outer(np.cos(th), 1 + 0 * ph)], -1)
    V = np.concatenate([[[0, 0, 1]], P.reshape(-1, 3), [[0, 0, -1]]])
    at = lambda i, j: 1 + i * nu + j % nu
    F = []
    for j in range(nu):
        F.append((0, at(0, j), at(0, j + 1)))
        F.append((len(V) - 1, at(nv - 2, j + 1), at(nv - 2, j)))
        for i in range(nv - 2):
            F += [(at(i, j), at(i + 1, j), at(i, j + 1)), (at(i, j + 1), at(i + 1, j), at(i + 1, j + 1))]
    return mg.Mesh(np.ascontiguousarray(V, np.float32), np.ascontiguousarray(F, np.int32), "poles")


@pytest.mark.parametrize("profile", ["ref", "mixed", "fp64"])
def test_long_rings_and_wide_cells(eng, oracle, profile):
    """Pole rings of 90 faces: more entries than a thread's list holds."""
    m = _poles()
    t = 2 * np.pi * np.arange(20) / 20
    cap = np.concatenate([[[0, 0, 1]], np.stack([0.1 * np.cos(t), 0.1 * np.sin(t), np.sqrt(0.99) + 0 * t], 1)])
    near = np.random.default_rng(1).normal(0, 0.02, (300, 3)) + np.array([[0, 0, 1], [0, 0, -1]]).repeat(150, 0)
    S0 = np.concatenate([cap, near, mg.sample_sites(m.V, m.F, 500, seed=2), [[0, 0, -1]]]).astype(np.float32)
    S, st = _run(eng, m, S0, 24, 0, 6, profile)
    r = oracle.lloyd_run(m.V, m.F, S0, 24, 0, 6, profile=oracle.PROFILES[profile])
    assert np.array_equal(st["knnv"], r["knnv"])
    assert np.array_equal(S, r["S"])


@pytest.mark.parametrize("kind", ["lattice", "mirrored", "repeated"])
@pytest.mark.parametrize("k,mode,profile,reuse", [(24, 1, "mixed", True), (8, 0, "ref", True), (20, 2, "fp64", True),
                                                  (20, 1, "ref", False)])
def test_equal_distances(eng, oracle, kind, k, mode, profile, reuse):
    """Sites on vertices and edges: faces at the same distance, the first of
    the rings' order wins."""
    m, S0 = order._sites(kind)
    S, st = _run(eng, m, S0, k, mode, 10, profile, reuse)
    r = oracle.lloyd_run(m.V, m.F, S0, k, mode, 10, profile=oracle.PROFILES[profile])
    assert np.array_equal(st["knn"], r["knn"]) and np.array_equal(st["knnv"], r["knnv"])
    assert np.array_equal(S, r["S"])


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("profile", ["ref", "mixed", "fp64"])
def test_freezing(eng, oracle, profile, mode):
    m = mg.torus(1.0, 0.3, 80, 40, noise_sigma=0.002, seed=3)
    S0 = mg.sample_sites(m.V, m.F, 1200, seed=4)
    S, st = _run(eng, m, S0, 20, mode, 40, profile)
    r = oracle.lloyd_run(m.V, m.F, S0, 20, mode, 40, profile=oracle.PROFILES[profile])
    assert r["frozen"].sum() > 100
    assert np.array_equal(st["frozen"], r["frozen"]) and np.array_equal(st["tier"], r["tier"])
    assert np.array_equal(S, r["S"])


@pytest.mark.parametrize("profile", ["ref", "mixed", "fp64"])
def test_open_cells_with_short_lists(eng, oracle, profile):
    """K = 8 and few sites: cells stay open, their centroids' vertex search is
    deferred."""
    m = mg.icosphere(5)
    S0 = mg.sample_sites(m.V, m.F, 150, seed=4)
    S, st = _run(eng, m, S0, 8, 0, 12, profile)
    r = oracle.lloyd_run(m.V, m.F, S0, 8, 0, 12, profile=oracle.PROFILES[profile])
    assert np.array_equal(st["knnv"], r["knnv"])
    assert np.array_equal(S, r["S"])


@pytest.mark.parametrize("profile", ["ref", "mixed", "fp64"])
def test_projection_shapes(eng, oracle, profile):
    m = mg.torus(1.0, 0.3, 60, 30, noise_sigma=0.002, seed=1)
    S0 = mg.sample_sites(m.V, m.F, 1500, seed=1)
    r = oracle.lloyd_run(m.V, m.F, S0, 24, 1, 12, profile=oracle.PROFILES[profile])
    for pb in (64, 128, 256):
        S, _ = _run(eng, m, S0, 24, 1, 12, profile, proj_block=pb)
        assert np.array_equal(S, r["S"])
