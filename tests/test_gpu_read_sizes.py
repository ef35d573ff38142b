"""Reads of sites and state on both sides of the sizes at which the host takes
over: the same values, and those of a device output."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("profile,n", [("mixed", 1), ("mixed", 8192), ("mixed", 8193), ("ref", 8886), ("ref", 8887),
                                       ("fp64", 4096), ("fp64", 4097), ("fp64", 9001)])
@pytest.mark.parametrize("reuse", [True, False])
def test_reads(oracle, profile, n, reuse):
    from gpu_cvt_b200 import engine as eng
    m = mg.icosphere(4)
    M = eng.Mesh(m.V, m.F)
    S0 = mg.sample_sites(m.V, m.F, n, seed=n)
    e = eng.Engine(eng.params(k=24, mode=1, profile=profile, knn_reuse=reuse), 1, n, eng.grid_cells(M, n, 24))
    g = e.add(M, S0)
    assert np.array_equal(e.sites(g), S0)
    e.run(3)
    S, st = e.sites(g), e.state(g)
    dev = torch.zeros((n, 3), device="cuda")
    e.sites_to_device(g, dev)
    assert np.array_equal(dev.cpu().numpy(), S, equal_nan=True)
    if profile == "fp64":
        assert np.array_equal(e.sites_f64(g).astype(np.float32), S)
    r = oracle.lloyd_run(m.V, m.F, S0, 24, 1, 3, profile=oracle.PROFILES[profile])
    assert np.array_equal(S, r["S"].astype(np.float32), equal_nan=True)
    if n > 24:
        for k in ("knn", "knnv", "frozen", "tier"):
            assert np.array_equal(st[k], r[k]), k
    e.close()
    M.close()
