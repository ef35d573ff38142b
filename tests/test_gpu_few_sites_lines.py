"""Both sides of the site counts at which the vertex search and the projection
change from 8 lanes to one thread per site, by profile."""
import numpy as np
import pytest

import test_gpu_site_order as order
from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("profile,n", [("mixed", 25000), ("mixed", 25001), ("fp64", 22000), ("fp64", 22001)])
def test_lines(oracle, profile, n):
    from gpu_cvt_b200 import engine as eng
    m = mg.torus(1.0, 0.3, 400, 40, noise_sigma=0.002, seed=4)
    S0 = mg.sample_sites(m.V, m.F, n, seed=n)
    S, st, _ = order._run(eng, m, S0, 12, 1, 3, profile, True)
    r = oracle.lloyd_run(m.V, m.F, S0, 12, 1, 3, profile=oracle.PROFILES[profile])
    assert np.array_equal(st["knnv"], r["knnv"])
    assert np.array_equal(S, r["S"])
