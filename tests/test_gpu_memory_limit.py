"""A program that holds all device memory still reads sites and state, and
places and removes segments: these calls need no more of it."""
import ctypes as C

import numpy as np
import pytest

from gpu_cvt_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N = 1_000_000


def _fill():
    """Device memory in blocks down to 4 MB until none is left, and what the
    library's pool still has in engines down to 1 MB."""
    from gpu_cvt_b200 import _lib, engine as eng
    _lib.call("cvt_release_cached_memory")
    torch.cuda.empty_cache()
    held, size = [], 1 << 34
    while size >= 1 << 22:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size //= 2
    for n in (1_000_000, 100_000, 10_000):
        while True:
            try:
                held.append(eng.Engine(eng.params(k=8, profile="ref"), 1, n, n))
            except _lib.CvtError:
                break
    return held


@pytest.mark.parametrize("profile", ["mixed", "fp64"])
def test_reads_and_placing_with_no_memory_left(profile):
    from gpu_cvt_b200 import _lib, engine as eng, stages as st
    m = mg.torus(1.0, 0.3, 200, 100, noise_sigma=0.002, seed=1)
    M = eng.Mesh(m.V, m.F)
    A = mg.sample_sites(m.V, m.F, N, seed=1)
    B = mg.sample_sites(m.V, m.F, N // 2, seed=2)
    Bd = torch.from_numpy(B).cuda()
    cells = eng.grid_cells(M, N, 8) + eng.grid_cells(M, N // 2, 8)
    e = eng.Engine(eng.params(k=8, mode=1, profile=profile), 2, N + N // 2, cells)
    a = e.add(M, A)

    def all_of(seg):
        r = {"S": e.sites(seg), **e.state(seg)}
        if profile == "fp64":
            r["D"] = e.sites_f64(seg)
        return r

    e.run(1)
    b = e.add(M, Bd)
    first = all_of(b)                        # before its first iteration
    e.run(2)
    want = all_of(a), all_of(b)
    e.remove(b)
    knn = torch.zeros((N // 2, 8), dtype=torch.int32, device="cuda")
    st.run_knn_bitonic_hubs(N // 2, 8, None, Bd, knn, None)
    held = _fill()
    try:
        with pytest.raises(_lib.CvtError):   # there is indeed none left
            st.run_knn_bitonic_hubs(N // 2, 8, None, Bd, knn, None)
        for sites in (B, Bd):                # host and device arrays
            b = e.add(M, sites)
            got = all_of(b), all_of(a)
            for k in first:
                assert np.array_equal(got[0][k], first[k]), k
            for k in want[0]:
                assert np.array_equal(got[1][k], want[0][k]), k
            if sites is B:
                e.remove(b)
    finally:
        for h in held:
            if isinstance(h, eng.Engine):
                h.close()
        del h, held
        torch.cuda.empty_cache()
    e.run(2)                                 # the segment placed with no memory left runs as before
    got = all_of(b)
    for k in want[1]:
        assert np.array_equal(got[k], want[1][k]), k
    e.close()
    M.close()


def test_output_that_is_not_device_memory():
    from gpu_cvt_b200 import _lib, engine as eng
    m = mg.icosphere(3)
    M = eng.Mesh(m.V, m.F)
    S = mg.sample_sites(m.V, m.F, 300, seed=0)
    e = eng.Engine(eng.params(k=12, profile="ref"), 1, 300, eng.grid_cells(M, 300, 12))
    g = e.add(M, S)
    e.run(2)
    out = np.zeros((300, 3), np.float32)
    with pytest.raises(_lib.CvtError):
        _lib.call("cvt_engine_get_sites", e.handle, g, out.ctypes.data_as(C.c_void_p), 1, None)
    pinned = torch.zeros((300, 3)).pin_memory()
    e.sites_to_device(g, pinned)             # the device can write pinned host memory
    torch.cuda.synchronize()
    assert np.array_equal(pinned.numpy(), e.sites(g))
    dev = torch.zeros((300, 3), device="cuda")
    e.sites_to_device(g, dev)
    assert np.array_equal(dev.cpu().numpy(), e.sites(g))
    e.close()
    M.close()
