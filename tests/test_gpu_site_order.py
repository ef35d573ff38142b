"""The engine stores a segment's sites in cell order and checks its neighbour
lists with one thread per site; lists, ties and every result must be those of
the caller's order, at block and warp edges, with exact distance ties (lattice
sites, mirrored and repeated sites) and through removal and re-use of slots.
The oracle works in the caller's order; everything is compared bit for bit."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def eng():
    from gpu_cvt_b200 import engine
    assert torch.cuda.is_available()
    return engine


def _run(eng, m, S0, k, mode, iters, profile, reuse):
    mesh = eng.Mesh(m.V, m.F)
    e = eng.Engine(eng.params(k=k, mode=mode, profile=profile, knn_reuse=reuse), 1, len(S0), eng.grid_cells(mesh, len(S0), k))
    g = e.add(mesh, S0)
    e.run(iters)
    S = e.sites_f64(g) if profile == "fp64" else e.sites(g)
    st = e.state(g)
    reused = sum(e.stats(g, i)["knn_reused"] for i in range(iters))
    e.close()
    mesh.close()
    return S, st, reused


def _sites(kind):
    if kind == "lattice":            # the reference's own start: the vertices, no noise, many equal distances
        m = mg.torus(1.0, 0.3, 64, 32)
        return m, m.V.copy()
    if kind == "mirrored":           # mirrored exactly in every axis, shuffled
        m = mg.icosphere(4)
        S = mg.sample_sites(m.V, m.F, 120, seed=5)
        S = np.concatenate([S * np.array(s, np.float32) for s in
                            [(1, 1, 1), (-1, 1, 1), (1, -1, 1), (1, 1, -1), (-1, -1, 1), (1, -1, -1), (-1, 1, -1),
                             (-1, -1, -1)]])
        return m, np.ascontiguousarray(np.random.default_rng(0).permutation(S))
    m = mg.icosphere(4)              # every site three times
    S = mg.sample_sites(m.V, m.F, 230, seed=6)
    return m, np.ascontiguousarray(np.random.default_rng(1).permutation(np.concatenate([S, S, S])))


@pytest.mark.parametrize("kind", ["lattice", "mirrored", "repeated"])
@pytest.mark.parametrize("k,mode,profile,reuse", [(24, 1, "mixed", True), (8, 0, "ref", True), (32, 2, "ref", True),
                                                  (20, 1, "ref", False)])
def test_equal_distances_keep_the_callers_order(eng, oracle, kind, k, mode, profile, reuse):
    m, S0 = _sites(kind)
    iters = 10
    S, st, reused = _run(eng, m, S0, k, mode, iters, profile, reuse)
    r = oracle.lloyd_run(m.V, m.F, S0, k, mode, iters, profile=oracle.PROFILES[profile])
    assert np.array_equal(st["knn"], r["knn"])
    assert np.array_equal(st["frozen"], r["frozen"])
    assert np.array_equal(S, r["S"])
    if reuse and kind == "lattice":
        assert reused > 0            # the tied lists went through the check


@pytest.mark.parametrize("n", [1, 2, 31, 33, 63, 64, 65, 129, 257])
@pytest.mark.parametrize("profile", ["mixed", "fp64"])
def test_block_edges(eng, oracle, n, profile):
    """Fewer sites than neighbours, one warp, one block and one more."""
    m = mg.icosphere(3)
    S0 = mg.sample_sites(m.V, m.F, n, seed=n)
    S, st, _ = _run(eng, m, S0, 16, 0, 4, profile, True)
    r = oracle.lloyd_run(m.V, m.F, S0, 16, 0, 4, profile=oracle.PROFILES[profile])
    if n > 16:
        assert np.array_equal(st["knn"], r["knn"])
    assert np.array_equal(S, r["S"], equal_nan=True)


def test_slots_used_again(eng, oracle):
    """Segments of other sizes placed in slots that removed ones left, at both
    buffer parities: each equals its own run."""
    m = mg.torus(1.0, 0.3, 60, 30, noise_sigma=0.002, seed=1)
    mesh = eng.Mesh(m.V, m.F)
    sizes = [700, 1300, 450]
    S = [mg.sample_sites(m.V, m.F, n, seed=n) for n in sizes]
    cells = sum(eng.grid_cells(mesh, n, 12) for n in sizes)
    e = eng.Engine(eng.params(k=12, mode=1, profile="ref"), 3, sum(sizes), cells)
    a, b = e.add(mesh, S[0]), e.add(mesh, S[1])
    e.run(3)
    e.remove(a)
    c = e.add(mesh, S[2])
    e.run(2)
    e.remove(b)
    d = e.add(mesh, S[1])
    e.run(4)
    for g, s, it in ((c, 2, 6), (d, 1, 4)):
        r = oracle.lloyd_run(m.V, m.F, S[s], 12, 1, it)
        assert np.array_equal(e.sites(g), r["S"])
        assert np.array_equal(e.state(g)["knn"], r["knn"])
    e.close()
    mesh.close()


def test_launches_follow_the_occupied_slots(eng, oracle):
    """A large engine whose launches cover only the occupied slots: segments
    that arrive beyond the covered part, and departures that shrink it, leave
    every result as it is alone (graph replays on both sides of a change)."""
    m = mg.icosphere(4)
    mesh = eng.Mesh(m.V, m.F)
    e = eng.Engine(eng.params(k=12, mode=0, profile="ref"), 8, 2_000_000, 8_000_000)
    S = {n: mg.sample_sites(m.V, m.F, n, seed=n) for n in (300, 1024, 5000, 70)}
    done = {}
    for n in (300, 1024, 5000):      # 300 -> 1324 -> 6324 slots
        done[n] = [e.add(mesh, S[n]), 0]
        e.run(5)
        for v in done.values():
            v[1] += 5
    for n in (300, 1024, 5000):
        assert np.array_equal(e.sites(done[n][0]), oracle.lloyd_run(m.V, m.F, S[n], 12, 0, done[n][1])["S"])
    for n in (300, 1024, 5000):
        e.remove(done[n][0])
    g = e.add(mesh, S[70])           # back to the smallest extent
    e.run(6)
    assert np.array_equal(e.sites(g), oracle.lloyd_run(m.V, m.F, S[70], 12, 0, 6)["S"])
    e.close()
    mesh.close()


@pytest.mark.parametrize("profile", ["ref", "mixed", "fp64"])
def test_cells_beyond_the_buffer_and_long_rings(eng, oracle, profile):
    """Cells with more than 16 vertices (a ring of 20 sites around one: redone
    with the 64-vertex cap), square cells of lone sites, and a mesh whose pole
    vertices have rings of 90 faces (more entries than the projection's list
    holds)."""
    nu, nv = 90, 24
    th = np.pi * np.arange(1, nv) / nv
    ph = 2 * np.pi * np.arange(nu) / nu
    V = np.concatenate([[[0, 0, 1]], np.stack([np.sin(th)[:, None] * np.cos(ph), np.sin(th)[:, None] * np.sin(ph),
                                              np.cos(th)[:, None] + 0 * ph], -1).reshape(-1, 3), [[0, 0, -1]]])
    i, j = np.meshgrid(np.arange(nv - 2), np.arange(nu), indexing="ij")
    a, b = 1 + i * nu + j, 1 + i * nu + (j + 1) % nu
    ring = np.arange(nu)
    F = np.concatenate([np.stack([0 * ring, 1 + ring, 1 + (ring + 1) % nu], 1),
                        np.stack([a, a + nu, b], -1).reshape(-1, 3), np.stack([b, a + nu, b + nu], -1).reshape(-1, 3),
                        np.stack([0 * ring + len(V) - 1, 1 + (nv - 2) * nu + (ring + 1) % nu, 1 + (nv - 2) * nu + ring], 1)])
    m = mg.Mesh(np.ascontiguousarray(V, np.float32), np.ascontiguousarray(F, np.int32), "poles")
    t = 2 * np.pi * np.arange(20) / 20
    cap = np.concatenate([[[0, 0, 1]], np.stack([0.1 * np.cos(t), 0.1 * np.sin(t), np.sqrt(0.99) + 0 * t], 1)])
    S0 = np.concatenate([cap, mg.sample_sites(m.V, m.F, 500, seed=2), [[0, 0, -1]]]).astype(np.float32)
    S, st, _ = _run(eng, m, S0, 24, 0, 5, profile, True)
    r = oracle.lloyd_run(m.V, m.F, S0, 24, 0, 5, profile=oracle.PROFILES[profile])
    assert np.array_equal(S, r["S"])
    one = oracle.lloyd_run(m.V, m.F, S0[:21], 24, 0, 2, profile=oracle.PROFILES[profile])  # the 20-gon, with the square around it
    S, _, _ = _run(eng, m, S0[:21], 24, 0, 2, profile, True)
    assert np.array_equal(S, one["S"], equal_nan=True)


@pytest.mark.parametrize("n,k,profile", [(1500, 32, "mixed"), (9000, 32, "ref"), (9000, 8, "mixed"), (9000, 24, "fp64")])
def test_uneven_density_searches(eng, oracle, n, k, profile):
    """Full searches whose radius holds far more or fewer sites than expected:
    nine tenths of the sites packed into a small cap."""
    m = mg.icosphere(5)
    S = mg.sample_sites(m.V, m.F, 60 * n, seed=n)
    cap = S[S[:, 2] > 0.97][: n - n // 10]
    S0 = np.random.default_rng(3).permutation(np.concatenate([cap, S[: n - len(cap)]]))
    S, st, _ = _run(eng, m, S0, k, 0, 3, profile, True)
    r = oracle.lloyd_run(m.V, m.F, S0, k, 0, 3, profile=oracle.PROFILES[profile])
    assert np.array_equal(st["knn"], r["knn"])
    assert np.array_equal(S, r["S"])


@pytest.mark.parametrize("n", [32768, 32769])
@pytest.mark.parametrize("profile,mode", [("ref", 0), ("mixed", 1), ("fp64", 2)])
def test_lanes_and_threads_meet(eng, oracle, n, profile, mode):
    """The largest site set whose vertex search and projection run with lanes
    per site, and the smallest with one thread each (thin faces among the
    mesh's, which the projection never skips)."""
    m = mg.torus(1.0, 0.3, 400, 40, noise_sigma=0.002, seed=4)
    S0 = mg.sample_sites(m.V, m.F, n, seed=n)
    S, st, _ = _run(eng, m, S0, 12, mode, 3, profile, True)
    r = oracle.lloyd_run(m.V, m.F, S0, 12, mode, 3, profile=oracle.PROFILES[profile])
    assert np.array_equal(st["knnv"], r["knnv"])
    assert np.array_equal(S, r["S"])
