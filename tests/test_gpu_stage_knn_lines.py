"""The stage searches on both sides of the lines at which they change between
a warp per query, groups of 32 points and a thread per query: the exact
(distance, index) order."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,kk", [(9999, 1), (10000, 1), (19999, 5), (20000, 5), (31999, 9), (32000, 9), (49999, 10),
                                  (50000, 10), (49999, 32), (50000, 32), (29999, 33), (30000, 33), (30000, 40),
                                  (30000, 41), (129999, 41), (130000, 41), (130000, 64), (30000, 2), (40000, 6)])
def test_points(oracle, n, kk):
    from gpu_cvt_b200 import stages as st
    m = mg.torus(1.0, 0.3, 100, 50, noise_sigma=0.002, seed=1)
    P = mg.sample_sites(m.V, m.F, n, seed=n)
    P[::997] = np.nan
    knn = torch.zeros((n, kk), dtype=torch.int32, device="cuda")
    d = torch.zeros((n, kk), dtype=torch.float32, device="cuda")
    st.run_knn_bitonic_hubs(n, kk, None, torch.from_numpy(P).cuda(), knn, d)
    ek, ed = oracle.knn_points(P, kk)
    live = np.isfinite(P).all(1)
    assert np.array_equal(knn.cpu().numpy().view(np.uint32)[live], ek[live])
    assert np.array_equal(d.cpu().numpy()[live], ed[live])


@pytest.mark.parametrize("nq,k", [(22619, 1), (22620, 1), (22621, 9), (39454, 10), (39455, 10), (39456, 25), (39460, 64)])
def test_queries(oracle, nq, k):
    """1,000 points: 8,600 and 15,000 times 1000 ** 0.14."""
    from gpu_cvt_b200 import stages as st
    m = mg.torus(1.0, 0.3, 40, 25, noise_sigma=0.002, seed=1)
    Q = mg.sample_sites(m.V, m.F, nq, seed=nq)
    Q[::3] *= np.float32(1.2)
    out = torch.zeros((nq, k), dtype=torch.int32, device="cuda")
    st.knn_vertices_bruteforce_k(torch.from_numpy(m.V).cuda(), len(m.V), torch.from_numpy(Q).cuda(), nq, None, out, kproj=k)
    assert np.array_equal(out.cpu().numpy(), oracle.knn_vertices(m.V, Q, k))


def test_single_neighbour_of_many_points_is_no_slower():
    """The nearest of 55k points: a thread per point, at most as long as for
    five neighbours of 60k and far below a warp per point's time."""
    from gpu_cvt_b200 import stages as st
    m = mg.torus(1.0, 0.3, 200, 100, noise_sigma=0.002, seed=1)

    def ms(n, kk):
        P = torch.from_numpy(mg.sample_sites(m.V, m.F, n, seed=n)).cuda()
        knn = torch.zeros((n, kk), dtype=torch.int32, device="cuda")
        return min(st.run_knn_bitonic_hubs(n, kk, None, P, knn, None) for _ in range(20))

    assert ms(55000, 1) < 1.15 * ms(60001, 5)
