"""The BVH build switches from levels over all triangles to one block per
subtree of at most 2048 triangles, and the traversals read a packed copy:
trees on both sides of the switch equal the recursive build node for node
(lattice meshes: many equal centroid coordinates, so the order must be that of
a stable sort), and distances equal a scan of every triangle."""
import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 8, 9, 17, 1024, 1025, 2047, 2048, 2049, 4096, 4099, 9001])
def test_trees_of_all_sizes(oracle, n):
    from gpu_cvt_b200.engine import Mesh
    m = mg.torus(1.0, 0.3, 96, 48)
    F = np.ascontiguousarray(m.F[:n])
    M = Mesh(m.V, F)
    nodes, tri = M.bvh()
    en, et = oracle.bvh_build(m.V, F)
    assert nodes.shape == en.shape and np.array_equal(tri, et)
    for f in en.dtype.names:
        assert np.array_equal(nodes[f], en[f]), f
    # one-sided distance of a shifted copy's probes, against the oracle's
    W = np.ascontiguousarray(m.V + np.float32([0.01, -0.02, 0.015]))
    d = M.hausdorff_from(torch.from_numpy(W).cuda(), torch.from_numpy(F).cuda())
    e = oracle.hausdorff_one_sided(W, F, m.V, F)
    assert abs(d - e) <= 1e-6 * e
    M.close()
