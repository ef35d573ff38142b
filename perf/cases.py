"""The timed workloads of the framework: what its users have it do, each
through the public entry point they call.

``listed()``   the workloads, ``draw(rng)`` another one of the same ranges;
``prepare``    what a program holds before the call, made from a seed;
``run``        one pass through the entry point, with its outputs;
``work``       the bytes and operations a pass cannot do without;
``exact``      the same outputs from plain FP64 torch, where they have such a
               value (one Lloyd step, FP64 runs of a few steps, distances).
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import math

import numpy as np
import torch

from gpu_cvt_b200 import _lib
from gpu_cvt_b200 import engine as E
from gpu_cvt_b200 import meshgen as mg
from gpu_cvt_b200 import server as SV
from gpu_cvt_b200 import stages as ST

SUPPORTED_K = (8, 12, 16, 20, 24, 32)


def listed():
    return [
        # a driver written against the reference's stage functions: one Lloyd step of a small
        # mesh (launch latency counts), and of a production-sized one in the mixed profile
        dict(name="stages_2k", kind="stages", shape="icosphere", tris=20_480, sites=2_000, k=20, profile="ref", mode=1),
        dict(name="stages_100k", kind="stages", shape="torus", tris=40_000, sites=100_000, k=24, profile="mixed", mode=2),
        # the neighbour search alone on a large point set (self + 32 neighbours)
        dict(name="knn_1m", kind="knn", shape="box", tris=500_000, sites=1_000_000, k=33),
        # one-call remesh with host arrays: the small plain configuration (latency), and the
        # 100k-site noisy torus with freezing, 100 iterations
        dict(name="remesh_2k", kind="remesh", shape="icosphere", tris=20_480, sites=2_000, k=20, profile="ref", mode=0,
             iters=50),
        dict(name="remesh_torus_100k", kind="remesh", shape="torus", tris=40_000, sites=100_000, k=24, profile="mixed",
             mode=1, iters=100),
        # many meshes of uneven size in one call, host arrays in and out, freezing off
        dict(name="batch_32", kind="batch", meshes=32, tri_lo=5_000, tri_hi=200_000, site_lo=1_000, site_hi=50_000, k=24,
             profile="mixed", mode=0, iters=100),
        # a resident mesh and engine: the largest site set, K=32, freezing on
        dict(name="engine_1m", kind="engine", shape="box", tris=500_000, sites=1_000_000, k=32, profile="mixed", mode=1,
             iters=25, proj="onering", frame="vertex"),
        # the FP64 profile (accuracy studies)
        dict(name="engine_fp64_30k", kind="engine", shape="torus", tris=20_000, sites=30_011, k=16, profile="fp64", mode=0,
             iters=5, proj="onering", frame="vertex"),
        # exact projection through the BVH and PCA frames
        dict(name="engine_bvh_pca_50k", kind="engine", shape="torus", tris=40_000, sites=50_000, k=24, profile="mixed",
             mode=2, iters=20, proj="bvh", frame="pca"),
        # a burst of requests through the server: device sampling, continuous batching, stop rules
        dict(name="serve_16", kind="serve", meshes=4, requests=16, tri_lo=20_000, tri_hi=200_000, site_lo=2_000,
             site_hi=200_000, k=24, profile="mixed", mode=1, iters=60),
        # the evaluation after a remesh: dual triangles, quality, Hausdorff distance
        dict(name="evaluate_100k", kind="evaluate", shape="torus", tris=40_000, sites=100_000, k=24, profile="mixed", mode=0,
             iters=8),
        # two meshes loaded from host arrays and compared (symmetric Hausdorff distance)
        dict(name="compare_200k", kind="compare", shape="box", tris=200_000, sites=0),
    ]


def draw(rng):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["stages", "stages", "knn", "remesh", "remesh", "batch", "engine", "engine", "engine", "serve",
                       "evaluate", "compare"])
    shape = rng.choice(["icosphere", "torus", "box", "family"])
    k = rng.choice(SUPPORTED_K)
    profile = rng.choice(["ref", "mixed", "mixed"])
    mode = rng.choice([0, 1, 2])
    tris = logu(5_000, 200_000)
    if kind == "stages":
        return dict(kind=kind, shape=shape, tris=tris, sites=logu(1_000, 200_000), k=k, profile=profile, mode=rng.choice([1, 2]))
    if kind == "knn":
        return dict(kind=kind, shape=shape, tris=tris, sites=logu(1_000, 1_000_000), k=rng.choice([6, 9, 17, 21, 25, 33, 48]))
    if kind == "remesh":
        return dict(kind=kind, shape=shape, tris=tris, sites=logu(1_000, 100_000), k=k, profile=profile, mode=mode,
                    iters=rng.randint(20, 100))
    if kind == "batch":
        return dict(kind=kind, meshes=rng.randint(8, 32), tri_lo=5_000, tri_hi=200_000, site_lo=1_000, site_hi=50_000,
                    k=rng.choice([16, 20, 24]), profile=profile, mode=mode, iters=rng.randint(30, 100))
    if kind == "engine":
        prof = rng.choice(["ref", "mixed", "mixed", "fp64"])
        return dict(kind=kind, shape=shape, tris=tris, sites=logu(2_000, 1_000_000 if prof != "fp64" else 200_000), k=k,
                    profile=prof, mode=mode, iters=rng.randint(3, 20), proj=rng.choice(["onering", "onering", "bvh"]),
                    frame=rng.choice(["vertex", "vertex", "pca"]))
    if kind == "serve":
        return dict(kind=kind, meshes=rng.randint(2, 6), requests=rng.randint(6, 16), tri_lo=20_000, tri_hi=200_000,
                    site_lo=2_000, site_hi=200_000, k=rng.choice([16, 20, 24]), profile=profile, mode=mode,
                    iters=rng.randint(20, 60))
    if kind == "evaluate":
        return dict(kind=kind, shape=shape, tris=tris, sites=logu(2_000, 200_000), k=k, profile=profile, mode=mode, iters=8)
    return dict(kind=kind, shape=shape, tris=tris, sites=0)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _mesh(shape, tris, seed):
    """Procedural mesh of about `tris` triangles; the seed sets its noise,
    size and proportions."""
    rng = np.random.default_rng(seed)
    if shape == "icosphere":
        return mg.icosphere(max(1, round(math.log(tris / 20.0, 4))), radius=float(rng.uniform(0.9, 1.1)))
    if shape == "torus":
        nv = max(8, round(math.sqrt(tris / 4.0)))
        return mg.torus(1.0, float(rng.uniform(0.28, 0.32)), max(8, round(tris / (2.0 * nv))), nv, 0.002, seed)
    if shape == "box":
        return mg.superellipsoid(float(rng.uniform(7.5, 8.5)), tris, 0.01, 1e-3, seed=seed)
    return mg.procedural_family(rng, max(1_000, tris // 2), tris)


def _cuda(a):
    return torch.from_numpy(a).cuda()


def _csr(V, F):
    """Vertex -> face lists in face order (offsets, faces)."""
    v = F.reshape(-1)
    f = np.repeat(np.arange(F.shape[0], dtype=np.int64), 3)
    order = np.argsort(v, kind="stable")
    off = np.zeros(V.shape[0] + 1, np.int32)
    np.cumsum(np.bincount(v, minlength=V.shape[0]), out=off[1:])
    return off, f[order].astype(np.int32)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _spread(lo, hi, n, salt):
    """n sizes spread evenly over the logarithm of [lo, hi], shuffled; the
    same for every seed."""
    x = np.exp(math.log(lo) + (np.arange(n) + 0.5) / n * math.log(hi / lo))
    return [int(round(v)) for v in np.random.default_rng(salt).permutation(x)]


def _batch_meshes(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for t, n in zip(_spread(case["tri_lo"], case["tri_hi"], case["meshes"], 1),
                    _spread(case["site_lo"], case["site_hi"], case["meshes"], 2)):
        m = mg.procedural_family(rng, t, t)
        out.append((m.V, m.F, mg.sample_sites(m.V, m.F, n, seed=int(rng.integers(0, 2**31 - 1)))))
    return out


def _inputs(case, seed):
    m = _mesh(case["shape"], case["tris"], seed)
    S = mg.sample_sites(m.V, m.F, case["sites"], seed=seed + 1) if case["sites"] else None
    return m, S


def _params(case):
    return E.params(k=case["k"], mode=case["mode"], profile=case["profile"], proj=case.get("proj", "onering"),
                    frame=case.get("frame", "vertex"))


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        ms = _batch_meshes(case, seed)
        pin = [[torch.from_numpy(a).pin_memory() for a in t] for t in ms]
        st.update(V=[p[0] for p in pin], F=[p[1] for p in pin], S=[p[2] for p in pin], prm=_params(case),
                  outs=[torch.empty_like(p[2]).pin_memory() for p in pin])
        return st
    if kind == "serve":
        rng = np.random.default_rng(seed)
        meshes = [mg.procedural_family(rng, t, t) for t in _spread(case["tri_lo"], case["tri_hi"], case["meshes"], 1)]
        st["requests"] = [SV.Request(i, int(rng.integers(0, case["meshes"])), n, int(rng.integers(0, 2**62)), 0.0)
                          for i, n in enumerate(_spread(case["site_lo"], case["site_hi"], case["requests"], 2))]
        st["server"] = SV.RemeshServer([(m.V, m.F) for m in meshes], k=case["k"], mode=case["mode"],
                                       profile=case["profile"], max_iters=case["iters"], keep_results=True)
        return st
    m, S = _inputs(case, seed)
    if kind == "compare":
        # the second mesh: the first with its vertices moved a little, one vertex in 100 a little more
        rng = np.random.default_rng(seed + 2)
        W = m.V + rng.normal(0.0, 1e-4, m.V.shape).astype(np.float32)
        far = rng.random(m.nV) < 0.01
        W[far] += rng.normal(0.0, 1e-3, (int(far.sum()), 3)).astype(np.float32)
        st.update(V=m.V, F=m.F, W=W)
        return st
    if kind == "remesh":
        st.update(V=m.V, F=m.F, S=S, prm=_params(case))
        return st
    if kind == "knn":
        n, k = case["sites"], case["k"]
        st.update(S=_cuda(S), knn=torch.empty((n, k), dtype=torch.int32, device="cuda"),
                  dist=torch.empty((n, k), dtype=torch.float32, device="cuda"))
        return st
    if kind == "stages":
        n, k = case["sites"], case["k"]
        off, fcs = _csr(m.V, m.F)

        def new(*shape, dtype=torch.float32):
            return torch.zeros(shape, dtype=dtype, device="cuda")

        st.update(R=mg.bbox_max_edge(m.V), V=_cuda(m.V), F=_cuda(m.F), off=_cuda(off), fcs=_cuda(fcs), S=_cuda(S),
                  N=new(m.nV, 3), knn1=new(n, k + 1, dtype=torch.int32), dist=new(n, k + 1),
                  knn=new(n, k, dtype=torch.int32), nv=new(n, 5, dtype=torch.int32), cv=new(n, 5, dtype=torch.int32),
                  U=new(n, 3), W=new(n, 3), cent=new(n, 3), nverts=new(n, dtype=torch.int32), Snew=new(n, 3),
                  tier=new(n, dtype=torch.uint8), streak=new(n, dtype=torch.uint8), cand=new(n, dtype=torch.uint8),
                  frozen=new(n, dtype=torch.uint8), counts=new(4, dtype=torch.int32), nsum=new(1, dtype=torch.int32))
        ST.vertex_normals(st["V"], st["F"], st["off"], st["fcs"], st["N"])
        return st
    # a resident mesh and an engine sized for the site set
    mesh = E.Mesh(m.V, m.F)
    n = case["sites"]
    eng = E.Engine(_params(case), 1, n, E.grid_cells(mesh, n, case["k"]))
    st.update(mesh=mesh, engine=eng, S=_cuda(S), out=torch.empty((n, 3), dtype=torch.float32, device="cuda"))
    if kind == "evaluate":
        st["seg"] = eng.add(mesh, st["S"], _stream())
        eng.run(case["iters"], _stream())
        st["faces"] = np.full((4 * n + 64, 3), -1, np.int32)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    return _RUN[case["kind"]](st, case)


def _run_stages(st, case):
    n, k, prof = case["sites"], case["k"], E.PROFILE[case["profile"]]
    nV, nF = st["V"].shape[0], st["F"].shape[0]
    thr2 = ((0.01 * st["R"]) * 0.01) * st["R"]
    ST.run_knn_bitonic_hubs(n, k + 1, None, st["S"], st["knn1"], st["dist"])
    ST.knn_drop_self(st["knn1"], st["knn"], n, k + 1, k)
    ST.knn_vertices_bruteforce_k(st["V"], nV, st["S"], n, None, st["nv"])
    ST.uv_from_nearest_vertex_normal(st["N"], st["nv"], st["U"], st["W"])
    ST.tier_ids(case["mode"], st["N"][st["nv"][:, 0].long()], st["knn"], st["tier"])
    ST.centroids_tangent_voronoi(st["S"], st["U"], st["W"], st["knn"], n, k, st["R"], st["cent"], prof, st["nverts"])
    ST.knn_vertices_bruteforce_k(st["V"], nV, st["cent"], n, None, st["cv"])
    ST.project_centroids_to_mesh(st["cent"], st["V"], st["F"], st["off"], st["fcs"], st["cv"], nV, nF, n, st["S"],
                                 st["Snew"], profile=prof)
    st["counts"].zero_()
    ST.freeze_test_streak(st["S"], st["Snew"], st["knn"], st["knn"], k, False, thr2, 4, st["streak"], st["cand"],
                          st["frozen"], st["counts"], st["tier"])
    st["nsum"].zero_()
    ST.count_frozen(st["frozen"], n, st["nsum"])
    return {x: st[x] for x in ("knn1", "dist", "knn", "nv", "U", "W", "tier", "cent", "nverts", "cv", "Snew", "streak",
                               "frozen", "nsum")}


def _run_knn(st, case):
    ST.run_knn_bitonic_hubs(case["sites"], case["k"], None, st["S"], st["knn"], st["dist"])
    return {"knn": st["knn"], "dist": st["dist"]}


def _run_remesh(st, case):
    out, counts = E.remesh(st["V"], st["F"], st["S"], iters=case["iters"], prm=st["prm"], with_counts=True)
    return {"sites": out, "counts": counts}


def _run_batch(st, case):
    return E.remesh_batch(st["V"], st["F"], st["S"], st["prm"], case["iters"], outs=st["outs"])


def _run_engine(st, case):
    eng, sp = st["engine"], _stream()
    seg = eng.add(st["mesh"], st["S"], sp)
    eng.run(case["iters"], sp)
    if case["profile"] == "fp64":
        out = eng.sites_f64(seg)
    else:
        eng.sites_to_device(seg, st["out"], sp)
        out = st["out"]
    s = eng.stats(seg, case["iters"] - 1)
    eng.remove(seg)
    return {"sites": out, "counts": [s["same"], s["low"], s["both"], s["newly_frozen"]], "max_motion": s["max_motion"]}


def _run_serve(st, case):
    reqs = [dataclasses.replace(r) for r in st["requests"]]
    st["server"].run(reqs)
    return {"sites": [r.result for r in reqs], "iters": [r.iters for r in reqs]}


def _run_evaluate(st, case):
    F, nf, o = st["faces"], C.c_int(), _lib.EvalOut()
    _lib.call("cvt_engine_faces", st["engine"].handle, st["seg"], F.ctypes.data_as(C.c_void_p), F.shape[0], C.byref(nf),
              C.byref(o), _stream())
    return {"faces": F, **{x: getattr(o, x) for x in ("dH", "Qmin", "Qavg", "theta_min", "theta_min_avg",
                                                      "theta_lt_30_pct", "theta_gt_90_pct", "n_faces")}}


def _run_compare(st, case):
    a, b = E.Mesh(st["V"], st["F"]), E.Mesh(st["W"], st["F"])
    d = a.hausdorff(b)
    r = {"dH": d["dH"], "ab": d["self_to_other"], "ba": d["other_to_self"], "R": b.R, "area": b.area, "diag": b.diag}
    a.close()
    b.close()
    return r


_RUN = dict(stages=_run_stages, knn=_run_knn, remesh=_run_remesh, batch=_run_batch, engine=_run_engine, serve=_run_serve,
            evaluate=_run_evaluate, compare=_run_compare)


# ---------------------------------------------------------------------------
# bytes and operations of a pass
# ---------------------------------------------------------------------------
def _site_flops(k):
    """One site, one Lloyd step: K distances (8) and bisectors (15), about six
    clips of a hexagon, a centroid, 5 + 1 vertex distances, six point-triangle
    tests."""
    return 23 * k + 6 * 60 + 60 + 6 * 8 + 6 * 70


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):  # means of the log-uniform sizes
        def mean(lo, hi):
            return (hi - lo) / math.log(hi / lo)
        items = case["meshes"] if kind == "batch" else case["requests"]
        n, t = items * mean(case["site_lo"], case["site_hi"]), case["meshes"] * mean(case["tri_lo"], case["tri_hi"])
        mesh_bytes = 18 * t  # 12 B per vertex (half as many as triangles), 12 B per face
        return {"bytes": mesh_bytes + 24 * n * case["iters"], "flops": n * case["iters"] * _site_flops(case["k"])}
    n, t = case["sites"], case["tris"]
    mesh_bytes = 18 * t
    if kind == "compare":
        # each of the 4.5 probes per face to a handful of triangles, both ways
        return {"bytes": 2 * mesh_bytes, "flops": 2 * 4.5 * t * 4 * 70}
    k = case["k"]
    if kind == "knn":
        return {"bytes": n * (12 + 8 * k), "flops": n * 8 * k}
    if kind == "stages":
        # site lists and distances, frames, centroids, vertex lists, projection, flags
        per = 12 + 8 * (k + 1) + 4 * k + 24 + 12 + 4 + 40 + 12 + 4
        return {"bytes": mesh_bytes + 6 * t + n * per, "flops": n * _site_flops(k)}
    if kind == "evaluate":
        return {"bytes": mesh_bytes + n * (12 + 4 * k) + 2 * n * 12, "flops": n * (_site_flops(k) + 11 * 4 * 70)}
    return {"bytes": mesh_bytes + 24 * n * case["iters"], "flops": n * case["iters"] * _site_flops(k)}


# ---------------------------------------------------------------------------
# the same in plain FP64
# ---------------------------------------------------------------------------
def _chunks(n, m):
    step = max(1, int(2e8) // max(m, 1))
    return [slice(i, min(n, i + step)) for i in range(0, n, step)]


def _nearest(P, Q, k, skip=None):
    """(distances squared, indices) of the k points of P nearest to each q,
    leaving out point skip[i] for query i."""
    ds, js = [], []
    for c in _chunks(Q.shape[0], P.shape[0]):
        q = Q[c]
        d = (q[:, None, 0] - P[None, :, 0]).square_()
        d += (q[:, None, 1] - P[None, :, 1]).square_()
        d += (q[:, None, 2] - P[None, :, 2]).square_()
        if skip is not None:
            rows = torch.nonzero(skip[c] < P.shape[0]).squeeze(1)
            d[rows, skip[c][rows]] = math.inf
        v, j = torch.topk(d, k, dim=1, largest=False, sorted=True)
        ds.append(v)
        js.append(j)
    return torch.cat(ds), torch.cat(js)


def _unit(x):
    return x / (x.square().sum(-1, keepdim=True) + 1e-30).sqrt()


def _vertex_normals(V, F):
    a, b, c = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    fn = torch.linalg.cross(b - a, c - a)
    N = torch.zeros_like(V)
    for j in range(3):
        N.index_add_(0, F[:, j], fn)
    return _unit(N)


def _frames(n):
    n = _unit(n)
    h = torch.zeros_like(n)
    flat = n[:, 2].abs() > 0.9
    h[flat, 0] = 1.0
    h[~flat, 2] = 1.0
    u = _unit(torch.linalg.cross(h, n))
    return u, _unit(torch.linalg.cross(n, u))


def _clip_centroid(S, U, W, knn, R):
    """Tangent-plane cell of every site, clipped by its listed neighbours'
    bisectors, and its area centroid in space."""
    n, cap = S.shape[0], 20
    poly = S.new_zeros(n, cap, 2)
    poly[:, :4] = torch.tensor([[-R, -R], [R, -R], [R, R], [-R, R]], dtype=S.dtype, device=S.device)
    cnt = torch.full((n,), 4, dtype=torch.long, device=S.device)
    at = torch.arange(cap, device=S.device)
    row = torch.arange(n, device=S.device)
    for t in range(knn.shape[1]):
        d = S[knn[:, t]] - S
        a, b, c = (d * U).sum(1), (d * W).sum(1), 0.5 * d.square().sum(1)
        f = a[:, None] * poly[..., 0] + b[:, None] * poly[..., 1] - c[:, None]
        here = at[None] < cnt[:, None]
        prev = torch.where(at[None] == 0, (cnt[:, None] - 1).clamp_min(0), at[None] - 1)
        ps, fs = poly.gather(1, prev[..., None].expand(-1, -1, 2)), f.gather(1, prev)
        ins_e, ins_s = f <= 0, fs <= 0
        cross = here & (ins_e != ins_s)
        keep = here & ins_e
        x = ps + (fs / (fs - f + 1e-300))[..., None] * (poly - ps)
        take = torch.stack([cross, keep], 2).reshape(n, -1)
        pts = torch.stack([x, poly], 2).reshape(n, -1, 2)
        pos = take.cumsum(1) - 1
        cnt = take.sum(1).clamp_max(cap)
        ok = take & (pos < cap)
        poly = torch.zeros_like(poly)
        poly[row[:, None].expand_as(pos)[ok], pos[ok]] = pts[ok]
    here = at[None] < cnt[:, None]
    nxt = torch.where(at[None] + 1 >= cnt[:, None], 0, at[None] + 1)
    q = poly.gather(1, nxt[..., None].expand(-1, -1, 2))
    cr = (poly[..., 0] * q[..., 1] - q[..., 0] * poly[..., 1]) * here
    c2 = ((poly + q) * cr[..., None]).sum(1) / (3.0 * cr.sum(1, keepdim=True))
    return S + U * c2[:, :1] + W * c2[:, 1:], cnt


def _closest(P, A, B, Cc):
    """Closest point of triangle (A, B, Cc) to P (broadcast over rows)."""
    def dot(x, y):
        return (x * y).sum(-1, keepdim=True)
    ab, ac, bc = B - A, Cc - A, Cc - B
    best, bd = None, None
    n = torch.linalg.cross(ab, ac)
    nn = dot(n, n)
    ap = P - A
    v = dot(torch.linalg.cross(ap, ac), n) / nn
    w = dot(torch.linalg.cross(ab, ap), n) / nn
    inside = (v >= 0) & (w >= 0) & (v + w <= 1)
    for o, e in ((A, ab), (A, ac), (B, bc)):
        p = o + e * (dot(P - o, e) / dot(e, e)).clamp(0, 1)
        d = dot(P - p, P - p)
        best, bd = (p, d) if best is None else (torch.where(d < bd, p, best), torch.minimum(d, bd))
    return torch.where(inside, A + ab * v + ac * w, best)


def _project(cent, V, F, off, fcs, cv):
    """Closest point over the one-rings of the listed vertices."""
    best = torch.full((cent.shape[0], 1), math.inf, dtype=cent.dtype, device=cent.device)
    out = cent.clone()
    for t in range(cv.shape[1]):
        lo, hi = off[cv[:, t]], off[cv[:, t] + 1]
        for e in range(int((hi - lo).max())):
            i = torch.nonzero(lo + e < hi).squeeze(1)
            f = F[fcs[lo[i] + e]]
            p = _closest(cent[i], V[f[:, 0]], V[f[:, 1]], V[f[:, 2]])
            d = (p - cent[i]).square().sum(1, keepdim=True)
            less = (d < best[i]).squeeze(1)
            best[i[less]], out[i[less]] = d[less], p[less]
    return out


def _step64(S, V, F, off, fcs, N, R, k, skip):
    d, j = _nearest(S, S, k + 1)
    me = torch.arange(S.shape[0], device=S.device)
    other = j != me[:, None]
    other &= other.cumsum(1) <= k
    knn = j[other].reshape(-1, k)
    nv = _nearest(V, S, 1)[1]
    U, W = _frames(N[nv[:, 0]])
    cent, cnt = _clip_centroid(S, U, W, knn, R)
    cv = _nearest(V, cent, 5, me if skip else None)[1]
    return dict(dist=d, U=U, W=W, cent=cent, Snew=_project(cent, V, F, off, fcs, cv))


def _hausdorff64(P, V, F):
    """Largest distance of the points P to the triangles."""
    A, B, Cc = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    far = P.new_zeros(())
    for c in _chunks(P.shape[0], 40 * F.shape[0]):
        q = _closest(P[c][:, None], A[None], B[None], Cc[None])
        far = torch.maximum(far, (q - P[c][:, None]).square().sum(-1).min(1).values.max())
    return float(far.sqrt())


def _probes(V, F):
    a, b, c = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    return torch.cat([V, (a + b + c) / 3, (a + b) / 2, (b + c) / 2, (c + a) / 2])


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def d64(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev).double()

    if kind == "compare":
        if case["tris"] > 40_000:  # every probe against every triangle
            return None
        st = prepare(case, seed)
        V, W, F = d64(st["V"]), d64(st["W"]), torch.from_numpy(st["F"]).to(dev).long()
        ab, ba = _hausdorff64(_probes(V, F), W, F), _hausdorff64(_probes(W, F), V, F)
        a, b, c = W[F[:, 0]], W[F[:, 1]], W[F[:, 2]]
        ext = W.max(0).values - W.min(0).values
        return {"dH": max(ab, ba), "ab": ab, "ba": ba, "R": float(ext.max()),
                "area": float(0.5 * torch.linalg.cross(b - a, c - a).norm(dim=1).sum()), "diag": float(ext.norm())}
    if kind not in ("stages", "knn", "engine") or case["sites"] > 150_000:
        return None
    if kind == "knn":
        S = d64(_inputs(case, seed)[1])
        return {"knn": None, "dist": _nearest(S, S, case["k"])[0]}
    plain = kind == "stages" or (case["profile"] == "fp64" and case["mode"] == 0 and case["iters"] <= 5 and
                                 case["proj"] == "onering" and case["frame"] == "vertex")
    if not plain or case["sites"] * (case["tris"] / 2 + case["sites"]) * case.get("iters", 1) > 4e10:
        return None
    m, S0 = _inputs(case, seed)
    off, fcs = (torch.from_numpy(a).to(dev).long() for a in _csr(m.V, m.F))
    S, V, F = d64(S0), d64(m.V), torch.from_numpy(m.F).to(dev).long()
    N, R, k = _vertex_normals(V, F), mg.bbox_max_edge(m.V), case["k"]
    if kind == "stages":
        r = _step64(S, V, F, off, fcs, N, R, k, False)
        return {x: r.get(x) for x in ("knn1", "dist", "knn", "nv", "U", "W", "tier", "cent", "nverts", "cv", "Snew",
                                      "streak", "frozen", "nsum")}
    # the run's own normals are FP32 (the mesh's): the frames differ by their rounding
    for _ in range(case["iters"]):
        before = S
        S = _step64(S, V, F, off, fcs, N, R, k, True)["Snew"]
    return {"sites": S.cpu().numpy(), "counts": None, "max_motion": float((S - before).norm(dim=1).max())}
