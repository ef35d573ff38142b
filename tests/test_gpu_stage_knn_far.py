"""Nearest-vertex queries off the surface, from one cell to far outside the
grid, on both sides and by both ways to begin (one thread or one warp per
query): rings while they are cheap, then one scan of all points; always the
exact (distance, index) order."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# in units of the radius of the unit sphere (a cell of 2,562 points: 0.1 for
# five neighbours, 0.2 for forty)
OFFSETS = np.array([0.0, 0.1, -0.1, 0.3, -0.3, 0.45, -0.45, 0.6, -0.6, 0.8, -0.9, -1.0, 1.5, 3.0, 30.0, 1e6])


@pytest.mark.parametrize("nq", [4001, 70001])
@pytest.mark.parametrize("k", [1, 5, 16, 40])
@pytest.mark.parametrize("ex", [False, True])
def test_offsets(oracle, nq, k, ex):
    from gpu_cvt_b200 import stages as st
    m = mg.icosphere(4)
    Q = mg.sample_sites(m.V, m.F, nq, seed=nq)
    Q = (Q * (1 + OFFSETS[np.arange(nq) % len(OFFSETS), None])).astype(np.float32)
    Q[::1000] = np.nan
    frozen = np.zeros(nq, np.uint8)
    frozen[3::11] = 1
    out = torch.full((nq, k), -7, dtype=torch.int32, device="cuda")
    st.knn_vertices_bruteforce_k(torch.from_numpy(m.V).cuda(), m.V.shape[0], torch.from_numpy(Q).cuda(), nq,
                                 torch.from_numpy(frozen).cuda(), out, kproj=k, exclude_self=ex)
    got, want = out.cpu().numpy(), oracle.knn_vertices(m.V, Q, k, exclude_self=ex)
    live = np.isfinite(Q).all(1) & (frozen == 0)
    assert np.array_equal(got[live], want[live])
    assert (got[frozen == 1] == -7).all()
    assert (got[~np.isfinite(Q).all(1) & (frozen == 0)] == -1).all()


def test_distances_too(oracle):
    """cvt_knn_query_to_points also writes the squared distances."""
    from gpu_cvt_b200 import stages as st
    m = mg.icosphere(4)
    nq, k = 70001, 7
    Q = mg.sample_sites(m.V, m.F, nq, seed=1)
    Q = (Q * (1 + OFFSETS[np.arange(nq) % len(OFFSETS), None])).astype(np.float32)
    knn = torch.zeros((nq, k), dtype=torch.int32, device="cuda")
    d = torch.zeros((nq, k), dtype=torch.float32, device="cuda")
    st.run_knn_bitonic_query_to_mesh(m.V.shape[0], torch.from_numpy(m.V).cuda(), torch.from_numpy(Q).cuda(), nq, k, None, knn, d)
    want = oracle.knn_vertices(m.V, Q, k)
    assert np.array_equal(knn.cpu().numpy(), want)
    e = Q[:, None, :] - m.V[want]
    assert np.allclose(d.cpu().numpy(), (e * e).sum(-1), rtol=1e-6)


def test_more_neighbours_than_points(oracle):
    from gpu_cvt_b200 import stages as st
    V = mg.sample_sites(mg.icosphere(2).V, mg.icosphere(2).F, 11, seed=0)
    for nq in (64, 70001):
        Q = np.random.default_rng(0).uniform(-3, 3, (nq, 3)).astype(np.float32)
        out = torch.zeros((nq, 16), dtype=torch.int32, device="cuda")
        st.knn_vertices_bruteforce_k(torch.from_numpy(V).cuda(), 11, torch.from_numpy(Q).cuda(), nq, None, out, kproj=16)
        assert np.array_equal(out.cpu().numpy(), oracle.knn_vertices(V, Q, 16))


def test_queries_some_cells_off_take_no_scans():
    """14 cells off 164k points: some times the surface's own queries, where a
    scan of all points per query takes a hundred times as long."""
    from gpu_cvt_b200 import stages as st
    m = mg.icosphere(7)
    V = torch.from_numpy(m.V).cuda()
    S = mg.sample_sites(m.V, m.F, 30000, seed=0)
    out = torch.zeros((30000, 5), dtype=torch.int32, device="cuda")

    def ms(Q):
        t = []
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            st.knn_vertices_bruteforce_k(V, V.shape[0], Q, 30000, None, out)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return min(t[1:])

    near = ms(torch.from_numpy(S).cuda())
    assert ms(torch.from_numpy(S * np.float32(1.17)).cuda()) < 25 * near
