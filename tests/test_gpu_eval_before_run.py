"""A segment that has not iterated yet has no neighbour lists: its evaluation
finds no dual triangles, whatever segment used its slots before."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("profile", ["mixed", "fp64"])
@pytest.mark.parametrize("reuse", [True, False])
@pytest.mark.parametrize("n_new", [900, 400])
def test_slots_of_a_removed_segment(profile, reuse, n_new):
    from gpu_cvt_b200 import engine as eng
    m = mg.icosphere(4)
    M = eng.Mesh(m.V, m.F)
    A = mg.sample_sites(m.V, m.F, 900, seed=1)
    B = mg.sample_sites(m.V, m.F, n_new, seed=2)

    def engine():
        return eng.Engine(eng.params(k=12, mode=1, profile=profile, knn_reuse=reuse), 1, 900, eng.grid_cells(M, 900, 12))

    e = engine()
    a = e.add(M, A)
    e.run(5)
    F, _ = e.faces(a)
    assert len(F) > 900                      # the lists that must not be read again
    e.remove(a)
    b = e.add(M, B)
    f = engine()
    g = f.add(M, B)
    got, want = e.faces(b), f.faces(g)
    assert len(got[0]) == 0
    assert np.array_equal(got[0], want[0])
    assert got[1] == want[1] and e.evaluate(b) == want[1]
    assert (e.state(b)["knn"] == 0).all()
    e.run(2)                                 # and from then on its own
    f.run(2)
    assert np.array_equal(e.faces(b)[0], f.faces(g)[0])
    e.close()
    f.close()
    M.close()
