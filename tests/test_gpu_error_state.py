"""A call that fails for lack of memory fails alone: the next one runs."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_call_after_a_failed_allocation(oracle):
    from gpu_cvt_b200 import _lib, engine as eng, stages as st
    m = mg.icosphere(3)
    S = mg.sample_sites(m.V, m.F, 500, seed=0)
    P = torch.from_numpy(S).cuda()
    knn = torch.zeros((500, 9), dtype=torch.int32, device="cuda")
    want = oracle.knn_points(S, 9)[0]
    M = eng.Mesh(m.V, m.F)
    for _ in range(2):
        with pytest.raises(_lib.CvtError) as ex:     # far more than the card has
            eng.Engine(eng.params(k=32), 1, 1_500_000_000, 2_000_000_000)
        assert ex.value.status == 3 or "memory" in str(ex.value)
        st.run_knn_bitonic_hubs(500, 9, None, P, knn, None)
        assert np.array_equal(knn.cpu().numpy().view(np.uint32), want)
        e = eng.Engine(eng.params(k=12), 1, 500, eng.grid_cells(M, 500, 12))
        g = e.add(M, S)
        e.run(2)
        assert np.isfinite(e.sites(g)).all()
        e.close()
    M.close()
