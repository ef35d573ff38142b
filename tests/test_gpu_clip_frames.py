"""The stage clip and the dual triangles take frames of any length and skew
from their caller: bit for bit the oracle's clip by all listed neighbours."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _case(oracle, frames, n=1500):
    m = mg.icosphere(4)
    S = mg.sample_sites(m.V, m.F, n, seed=2)
    N = (S / np.linalg.norm(S, axis=1, keepdims=True)).astype(np.float32)
    U, V = oracle.frames(N, np.arange(n))
    knn = oracle.drop_self(oracle.knn_points(S, 33)[0], 32)
    if frames == "unit":
        pass
    elif frames == "long":
        U, V = 3 * U, 3 * V
    elif frames == "short":
        U, V = 0.2 * U, 0.2 * V
    elif frames == "stretched":
        U = 5 * U
    elif frames == "skew":                   # nearly parallel unit vectors
        V = 0.95 * U + np.sqrt(1 - 0.95**2) * V
    elif frames == "tilted":                 # out of the tangent plane
        U, V = U + N, V - 2 * N
    elif frames == "mixed":                  # every site another length, some not finite
        f = np.random.default_rng(0).uniform(0.1, 8.0, (n, 1)).astype(np.float32)
        f[::50] = np.nan
        f[7::50] = np.inf
        with np.errstate(invalid="ignore"):
            U, V = f * U, V / f
    return S, np.ascontiguousarray(U, np.float32), np.ascontiguousarray(V, np.float32), knn


FRAMES = ["unit", "long", "short", "stretched", "skew", "tilted", "mixed"]


@pytest.mark.parametrize("frames", FRAMES)
@pytest.mark.parametrize("R", [2.0, 0.15])
@pytest.mark.parametrize("profile", [0, 1])
def test_clip(oracle, frames, R, profile):
    from gpu_cvt_b200 import stages as st
    S, U, V, knn = _case(oracle, frames)
    dev = lambda a: torch.from_numpy(a).cuda()
    cent = torch.zeros((len(S), 3), dtype=torch.float32, device="cuda")
    nv = torch.zeros(len(S), dtype=torch.int32, device="cuda")
    st.centroids_tangent_voronoi(dev(S), dev(U), dev(V), dev(knn.view(np.int32)), len(S), knn.shape[1], R, cent, profile, nv)
    co, nvo = oracle.clip_centroids(S, U, V, knn, R, profile=profile, return_nverts=True)
    assert np.array_equal(nv.cpu().numpy(), nvo)
    assert np.array_equal(cent.cpu().numpy(), co, equal_nan=True)


@pytest.mark.parametrize("frames", FRAMES)
def test_dual_triangles(oracle, frames):
    from gpu_cvt_b200 import stages as st
    S, U, V, knn = _case(oracle, frames)
    dev = lambda a: torch.from_numpy(a).cuda()
    R2 = float(mg.bbox_max_edge(S))
    F = st.extract_faces(dev(S), dev(U), dev(V), dev(knn.view(np.int32)), R2)
    assert np.array_equal(F.cpu().numpy(), oracle.extract_faces(S, U, V, knn, R2))
