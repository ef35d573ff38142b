"""The stage searches choose between one warp per query, groups of 32 points
and one thread per query by the number of queries and neighbours; all give the
exact (distance, index) order: on both sides of every switch, with equal
distances, packed and far-off points, frozen rows, non-finite points, and in
the allocation-free form."""
import ctypes as C

import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _points(kind, n, seed=0):
    rng = np.random.default_rng(seed)
    if kind == "surface":
        m = mg.torus(1.0, 0.3, 100, 50, noise_sigma=0.002, seed=1)
        return mg.sample_sites(m.V, m.F, n, seed=seed)
    if kind == "lattice":
        nu = int(np.ceil(np.sqrt(2 * n)))
        return np.ascontiguousarray(mg.torus(1.0, 0.3, nu, (n + nu - 1) // nu).V[:n])
    if kind == "packed":             # most points in one thousandth of the box, some repeated
        P = rng.normal(0.0, 1e-3, (n, 3))
        P[: n // 10] = rng.uniform(-1, 1, (n // 10, 3))
        P[n // 2: n // 2 + 50] = P[n // 2]
        return rng.permutation(P).astype(np.float32)
    P = rng.uniform(-1, 1, (n, 3)).astype(np.float32)  # a volume
    P[::97] = np.nan
    return P


@pytest.mark.parametrize("kind", ["surface", "lattice", "packed", "nan"])
@pytest.mark.parametrize("n,kk", [(40, 64), (3001, 25), (59999, 10), (60000, 10), (60001, 9), (70001, 33), (61000, 40),
                                  (60000, 41)])
def test_points(oracle, kind, n, kk):
    from gpu_cvt_b200 import _lib, stages as st
    P = _points(kind, n, seed=n + kk)
    ek, ed = oracle.knn_points(P, kk)
    T = torch.from_numpy(P).cuda()
    frozen = np.zeros(n, np.uint8)
    frozen[5::7] = 1
    for fz in (None, torch.from_numpy(frozen).cuda()):
        knn = torch.full((n, kk), -7, dtype=torch.int32, device="cuda")
        dist = torch.full((n, kk), -1.0, dtype=torch.float32, device="cuda")
        st.run_knn_bitonic_hubs(n, kk, fz, T, knn, dist)
        k, d = knn.cpu().numpy().view(np.uint32), dist.cpu().numpy()
        live = np.isfinite(P).all(1) if fz is None else np.isfinite(P).all(1) & (frozen == 0)
        assert np.array_equal(k[live], ek[live]) and np.array_equal(d[live], ed[live])
        if fz is not None:
            assert (k[frozen == 1] == np.uint32(2**32 - 7)).all()
    knn2 = torch.zeros_like(knn)
    _lib.call("cvt_knn_sites_noalloc", C.c_void_p(T.data_ptr()), n, kk, None, C.c_void_p(knn2.data_ptr()), None,
              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    live = np.isfinite(P).all(1)
    assert np.array_equal(knn2.cpu().numpy().view(np.uint32)[live], ek[live])


@pytest.mark.parametrize("nq", [300, 49999, 50000, 70007])
@pytest.mark.parametrize("ex", [False, True])
def test_far_queries(oracle, nq, ex):
    """Queries off the surface, some of them many cells away."""
    from gpu_cvt_b200 import stages as st
    m = mg.icosphere(4)
    rng = np.random.default_rng(nq)
    Q = mg.sample_sites(m.V, m.F, nq, seed=nq)
    far = rng.random(nq) < 0.01
    Q[far] *= rng.uniform(1.5, 30.0, (int(far.sum()), 1)).astype(np.float32)
    Q[~far] *= rng.uniform(0.9, 1.1, (int((~far).sum()), 1)).astype(np.float32)
    out = torch.zeros((nq, 5), dtype=torch.int32, device="cuda")
    st.knn_vertices_bruteforce_k(torch.from_numpy(m.V).cuda(), m.V.shape[0], torch.from_numpy(Q).cuda(), nq, None, out,
                                 exclude_self=ex)
    assert np.array_equal(out.cpu().numpy(), oracle.knn_vertices(m.V, Q, 5, exclude_self=ex))
