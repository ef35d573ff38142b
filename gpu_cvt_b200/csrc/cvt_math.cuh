// Device geometry for the tangent-plane CVT Lloyd step.
//
// Rounding is pinned: the library is compiled with -fmad=false, so a*b+c is
// two rounded operations unless an explicit fmaT() is written, and every
// division / square root is the IEEE-rounded intrinsic.  The operation order
// of each routine follows the reference kernels it replaces (cited below);
// the reference's rsqrtf() becomes 1/sqrt (IEEE), a <=1-ulp difference.
#pragma once
#include <climits>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cvt {

enum Profile { PROF_REF = 0, PROF_MIXED = 1, PROF_FP64 = 2 };

template <class T> struct V3 { T x, y, z; };
template <class T> struct V2 { T x, y; };

__device__ __forceinline__ float fmaT(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmaT(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float divT(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double divT(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float sqrtT(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double sqrtT(double a) { return __dsqrt_rn(a); }
__device__ __forceinline__ float absT(float a) { return fabsf(a); }
__device__ __forceinline__ double absT(double a) { return fabs(a); }
template <class T> __device__ __forceinline__ bool finiteT(T a) { return isfinite(a); }

template <class T> __device__ __forceinline__ V3<T> sub3(V3<T> a, V3<T> b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <class T> __device__ __forceinline__ T dot3(V3<T> a, V3<T> b) {
  return fmaT(a.z, b.z, fmaT(a.y, b.y, a.x * b.x));
}
template <class T> __device__ __forceinline__ V3<T> cross3(V3<T> a, V3<T> b) {
  return {fmaT(a.y, b.z, -(a.z * b.y)), fmaT(a.z, b.x, -(a.x * b.z)), fmaT(a.x, b.y, -(a.y * b.x))};
}
template <class T> __device__ __forceinline__ T dist2(V3<T> p, V3<T> q) {
  T dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
  return fmaT(dz, dz, fmaT(dy, dy, dx * dx));
}
template <class T, class S> __device__ __forceinline__ V3<T> cvt3(V3<S> a) { return {(T)a.x, (T)a.y, (T)a.z}; }
template <class T> __device__ __forceinline__ V3<T> ld3(const T* __restrict__ p, long i) {
  return {p[3 * i], p[3 * i + 1], p[3 * i + 2]};
}
template <class T> __device__ __forceinline__ void st3(T* __restrict__ p, long i, V3<T> v) {
  p[3 * i] = v.x; p[3 * i + 1] = v.y; p[3 * i + 2] = v.z;
}
template <class T> __device__ __forceinline__ bool finite3(V3<T> a) {
  return finiteT(a.x) && finiteT(a.y) && finiteT(a.z);
}

// --------------------------------------------------------------------------
// tangent frame from a vertex normal (site_normals.cuh:69-110)
// --------------------------------------------------------------------------
template <class T> struct Frame { V3<T> u, v; };

template <class T> __device__ __forceinline__ Frame<T> frame_from_normal(V3<T> n) {
  const T tiny = (T)1e-30;
  T inv = divT((T)1, sqrtT(dot3(n, n) + tiny));
  n = {n.x * inv, n.y * inv, n.z * inv};
  V3<T> h = (absT(n.z) > (T)0.9) ? V3<T>{1, 0, 0} : V3<T>{0, 0, 1};
  V3<T> u = cross3(h, n);
  T iu = divT((T)1, sqrtT(dot3(u, u) + tiny));
  u = {u.x * iu, u.y * iu, u.z * iu};
  V3<T> v = cross3(n, u);
  T iv = divT((T)1, sqrtT(dot3(v, v) + tiny));
  v = {v.x * iv, v.y * iv, v.z * iv};
  return {u, v};
}

// --------------------------------------------------------------------------
// PCA normal of a site's neighbourhood (frame option; the reference builds
// every frame from the nearest vertex normal, site_normals.cuh:69-110).
// The eigenvector of the smallest eigenvalue of the covariance C of the
// listed neighbours' offsets, found by power iteration on the adjugate of C,
// which has the same eigenvectors with the order reversed (error shrinks by
// l1 / l2 per step: fast wherever the neighbourhood is a surface patch, even
// a narrow one).  The iteration starts from the reference normal n0 and runs
// a fixed kPcaSteps steps; its sign is then chosen to agree with n0.  Fewer
// than 3 neighbours, a zero spread, or a non-finite result give n0 back.
// Only IEEE-rounded arithmetic with an explicit operation order, so a CPU
// restatement reproduces the bits.
// --------------------------------------------------------------------------
constexpr int kPcaSteps = 8;

template <class T, class NB>
__device__ __forceinline__ V3<T> pca_normal(const NB& nb, int K, V3<T> si, V3<T> n0) {
  T sx = 0, sy = 0, sz = 0, xx = 0, xy = 0, xz = 0, yy = 0, yz = 0, zz = 0;
  int m = 0;
  for (int t = 0; t < K; ++t) {
    const uint32_t j = nb.id(t);
    if (!nb.valid(j)) continue;
    const V3<T> d = sub3(nb.pos(j), si);
    sx = sx + d.x; sy = sy + d.y; sz = sz + d.z;
    xx = fmaT(d.x, d.x, xx); xy = fmaT(d.x, d.y, xy); xz = fmaT(d.x, d.z, xz);
    yy = fmaT(d.y, d.y, yy); yz = fmaT(d.y, d.z, yz); zz = fmaT(d.z, d.z, zz);
    ++m;
  }
  if (m < 3) return n0;
  const T im = divT((T)1, (T)m);
  const T mx = sx * im, my = sy * im, mz = sz * im;
  // C = sum d d^T - m mean mean^T = sum d d^T - s mean^T
  const T cxx = fmaT(-sx, mx, xx), cxy = fmaT(-sx, my, xy), cxz = fmaT(-sx, mz, xz);
  const T cyy = fmaT(-sy, my, yy), cyz = fmaT(-sy, mz, yz), czz = fmaT(-sz, mz, zz);
  const T tr = (cxx + cyy) + czz;
  if (!(tr > (T)1e-30)) return n0;
  // adjugate of C: eigenvalues l2 l3, l1 l3, l1 l2 for C's l1 <= l2 <= l3,
  // so the normal's (l1) direction dominates by the factor l2 / l1
  const T axx = fmaT(cyy, czz, -(cyz * cyz)), axy = fmaT(cxz, cyz, -(cxy * czz)), axz = fmaT(cxy, cyz, -(cxz * cyy));
  const T ayy = fmaT(cxx, czz, -(cxz * cxz)), ayz = fmaT(cxy, cxz, -(cxx * cyz)), azz = fmaT(cxx, cyy, -(cxy * cxy));
  V3<T> v = n0;
  for (int it = 0; it < kPcaSteps; ++it) {
    const V3<T> w{fmaT(axz, v.z, fmaT(axy, v.y, axx * v.x)), fmaT(ayz, v.z, fmaT(ayy, v.y, axy * v.x)),
                  fmaT(azz, v.z, fmaT(ayz, v.y, axz * v.x))};
    const T nw = sqrtT(dot3(w, w));
    if (!(nw > (T)1e-30)) return n0;
    const T inv = divT((T)1, nw);
    v = {w.x * inv, w.y * inv, w.z * inv};
  }
  if (!finite3(v)) return n0;
  if (dot3(v, n0) < (T)0) v = {-v.x, -v.y, -v.z};
  return v;
}

// --------------------------------------------------------------------------
// centroid of the clipped polygon (2dClip.cuh:55-80); Neumaier compensation
// in the MIXED profile.
// --------------------------------------------------------------------------
template <class T> struct CSum {
  T s, c;
  __device__ __forceinline__ CSum() : s(0), c(0) {}
  __device__ __forceinline__ void add(T x) {
    T t = s + x;
    if (absT(s) >= absT(x)) c += (s - t) + x; else c += (x - t) + s;
    s = t;
  }
  __device__ __forceinline__ T get() const { return s + c; }
};

// Polygon accessor: vertex k of the polygon currently held in a buffer.
template <class P, class Buf>
__device__ __forceinline__ V2<P> poly_centroid(const Buf& poly, int n, bool compensated) {
  const P nanv = (P)NAN;
  if (n < 3) return {nanv, nanv};
  P A2, Cx, Cy;
  if (!compensated) {
    A2 = 0; Cx = 0; Cy = 0;
    V2<P> p = poly.get(0);
    for (int i = 0; i < n; ++i) {
      V2<P> q = poly.get(i + 1 == n ? 0 : i + 1);
      P cr = fmaT(p.x, q.y, -(q.x * p.y));
      A2 = A2 + cr;
      Cx = fmaT(p.x + q.x, cr, Cx);
      Cy = fmaT(p.y + q.y, cr, Cy);
      p = q;
    }
  } else {
    CSum<P> a, x, y;
    V2<P> p = poly.get(0);
    for (int i = 0; i < n; ++i) {
      V2<P> q = poly.get(i + 1 == n ? 0 : i + 1);
      P cr = fmaT(p.x, q.y, -(q.x * p.y));
      a.add(cr);
      x.add((p.x + q.x) * cr);
      y.add((p.y + q.y) * cr);
      p = q;
    }
    A2 = a.get(); Cx = x.get(); Cy = y.get();
  }
  P A = (P)0.5 * A2;
  if (absT(A) < (P)1e-18) {
    P mx = 0, my = 0;
    for (int i = 0; i < n; ++i) { V2<P> q = poly.get(i); mx = mx + q.x; my = my + q.y; }
    return {divT(mx, (P)n), divT(my, (P)n)};
  }
  P inv6A = divT((P)1, (P)6 * A);
  return {Cx * inv6A, Cy * inv6A};
}

// --------------------------------------------------------------------------
// closest point on a triangle (near_project.cuh:12-53)
// --------------------------------------------------------------------------
template <class T> __device__ __forceinline__ V3<T> closest_point_tri(V3<T> P, V3<T> A, V3<T> B, V3<T> C) {
  const T e = (T)1e-30;
  V3<T> AB = sub3(B, A), AC = sub3(C, A), AP = sub3(P, A);
  T d1 = dot3(AB, AP), d2 = dot3(AC, AP);
  if (d1 <= 0 && d2 <= 0) return A;
  V3<T> BP = sub3(P, B);
  T d3 = dot3(AB, BP), d4 = dot3(AC, BP);
  if (d3 >= 0 && d4 <= d3) return B;
  T vc = fmaT(d1, d4, -(d3 * d2));
  if (vc <= 0 && d1 >= 0 && d3 <= 0) {
    T v = divT(d1, (d1 - d3) + e);
    return {fmaT(AB.x, v, A.x), fmaT(AB.y, v, A.y), fmaT(AB.z, v, A.z)};
  }
  V3<T> CP = sub3(P, C);
  T d5 = dot3(AB, CP), d6 = dot3(AC, CP);
  if (d6 >= 0 && d5 <= d6) return C;
  T vb = fmaT(d5, d2, -(d1 * d6));
  if (vb <= 0 && d2 >= 0 && d6 <= 0) {
    T w = divT(d2, (d2 - d6) + e);
    return {fmaT(AC.x, w, A.x), fmaT(AC.y, w, A.y), fmaT(AC.z, w, A.z)};
  }
  T va = fmaT(d3, d6, -(d5 * d4));
  if (va <= 0 && (d4 - d3) >= 0 && (d5 - d6) >= 0) {
    T w = divT(d4 - d3, ((d4 - d3) + (d5 - d6)) + e);
    V3<T> BC = sub3(C, B);
    return {fmaT(BC.x, w, B.x), fmaT(BC.y, w, B.y), fmaT(BC.z, w, B.z)};
  }
  T denom = divT((T)1, ((va + vb) + vc) + e);
  T v = vb * denom, w = vc * denom;
  return {A.x + fmaT(AB.x, v, AC.x * w), A.y + fmaT(AB.y, v, AC.y * w), A.z + fmaT(AB.z, v, AC.z * w)};
}

// closest point over the one-rings of the kproj nearest vertices
// (project_centroids_to_mesh, near_project.cuh:149-189).  Q is the
// arithmetic type (double for the MIXED barycentrics).  A face that contains
// an earlier listed vertex was already tested in that vertex's one-ring with
// the same inputs; a repeat can never pass the strict '<', so it is skipped.
template <class T, class Q>
__device__ __forceinline__ V3<T> project_onering(V3<T> c, const float* __restrict__ V, int nV,
                                                 const int* __restrict__ F, int nF,
                                                 const int* __restrict__ off, const int* __restrict__ fcs,
                                                 const int* knnv, int kproj) {
  V3<Q> cq = cvt3<Q>(c), bp = cq;
  Q best = (Q)1e30;
  for (int t = 0; t < kproj; ++t) {
    int v = knnv[t];
    if ((unsigned)v >= (unsigned)nV) continue;
    int beg = __ldg(off + v), end = __ldg(off + v + 1);
    for (int ii = beg; ii < end; ++ii) {
      int fi = __ldg(fcs + ii);
      if ((unsigned)fi >= (unsigned)nF) continue;
      int ia = __ldg(F + 3 * fi), ib = __ldg(F + 3 * fi + 1), ic = __ldg(F + 3 * fi + 2);
      bool seen = false;
      for (int s = 0; s < t; ++s) {
        const int w = knnv[s];
        seen = seen || w == ia || w == ib || w == ic;
      }
      if (seen) continue;
      V3<Q> A = {(Q)__ldg(V + 3 * ia), (Q)__ldg(V + 3 * ia + 1), (Q)__ldg(V + 3 * ia + 2)};
      V3<Q> B = {(Q)__ldg(V + 3 * ib), (Q)__ldg(V + 3 * ib + 1), (Q)__ldg(V + 3 * ib + 2)};
      V3<Q> C = {(Q)__ldg(V + 3 * ic), (Q)__ldg(V + 3 * ic + 1), (Q)__ldg(V + 3 * ic + 2)};
      V3<Q> p = closest_point_tri(cq, A, B, C);
      V3<Q> dd = sub3(p, cq);
      Q d2 = dot3(dd, dd);
      if (d2 < best) { best = d2; bp = p; }
    }
  }
  return cvt3<T>(bp);
}

// One-ring records: for every vertex->face CSR entry (same order as the CSR),
// a head and a body.  The head is the face's bounding sphere {centre, radius}
// (16 bytes, a ring of six is 96 contiguous bytes); the body is the face's
// three corner positions and vertex ids,
//   r0 = {A.x, A.y, A.z, B.x}, r1 = {B.y, B.z, C.x, C.y}, r2 = {C.z, ia, ib, ic}
// (ids as int bits).  A projection reads one offset and then the heads of the
// ring, and the body only of the faces that the sphere test keeps (about a
// third), instead of the chain CSR entry -> face -> corners.  The sphere is
// centred on the float-rounded centroid; its radius is the largest corner
// distance, computed in double and rounded up, so it holds the whole
// triangle.  radius < 0 marks a face the projection never skips: an invalid
// entry, or a triangle with a corner angle below ~5.7 degrees
// (sin^2 < kPruneSin2), whose face-region formula is ill-conditioned.
constexpr int kRingBody = 3;  // 16-byte words of a body
constexpr double kPruneSin2 = 0.01;

__global__ void k_build_ring_records(const float* __restrict__ V, const int* __restrict__ F, int nF,
                                     const int* __restrict__ fcs, long n_entries, float4* __restrict__ head,
                                     float4* __restrict__ body) {
  const long ii = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ii >= n_entries) return;
  const int fi = fcs[ii];
  int ia = -1, ib = -1, ic = -1;
  float a[3] = {0.f, 0.f, 0.f}, b[3] = {0.f, 0.f, 0.f}, c[3] = {0.f, 0.f, 0.f};
  float4 sph = make_float4(0.f, 0.f, 0.f, -1.f);
  if ((unsigned)fi < (unsigned)nF) {
    ia = F[3 * fi]; ib = F[3 * fi + 1]; ic = F[3 * fi + 2];
    for (int k = 0; k < 3; ++k) { a[k] = V[3 * ia + k]; b[k] = V[3 * ib + k]; c[k] = V[3 * ic + k]; }
    float m[3];
    double r2 = 0.0;
    for (int k = 0; k < 3; ++k) m[k] = (float)(((double)a[k] + (double)b[k] + (double)c[k]) / 3.0);
    const float* P[3] = {a, b, c};
    bool ok = true;
    for (int j = 0; j < 3; ++j) {
      double d2 = 0.0, u[3], v[3];
      for (int k = 0; k < 3; ++k) {
        const double d = (double)P[j][k] - (double)m[k];
        d2 += d * d;
        u[k] = (double)P[(j + 1) % 3][k] - (double)P[j][k];
        v[k] = (double)P[(j + 2) % 3][k] - (double)P[j][k];
      }
      r2 = fmax(r2, d2);
      const double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2], cz = u[0] * v[1] - u[1] * v[0];
      const double uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2], vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
      ok = ok && (cx * cx + cy * cy + cz * cz) >= kPruneSin2 * (uu * vv);  // false for NaN / zero-length edges
    }
    const float rad = __double2float_ru(sqrt(r2) * (1.0 + 1e-9));
    if (ok && isfinite(rad)) sph = make_float4(m[0], m[1], m[2], rad);
  }
  body[kRingBody * ii] = make_float4(a[0], a[1], a[2], b[0]);
  body[kRingBody * ii + 1] = make_float4(b[1], b[2], c[0], c[1]);
  body[kRingBody * ii + 2] = make_float4(c[2], __int_as_float(ia), __int_as_float(ib), __int_as_float(ic));
  head[ii] = sph;
}

// project_onering over the one-ring records, for the five nearest vertices:
// the same result bit for bit, from the few faces that can hold it.
//
// Whatever the closest-point code returns for a face lies at a distance from
// c between lb and ub,
//   lb = |c - centre| - radius - E,  ub = |c - centre| + E,
//   E  = 0.05 (|c - centre| + radius) + 1e-4 max|coordinate|
//        + 1e-4 |c - centre|^2 / radius
// (the centre is the face's centroid up to rounding).  E is far above the
// rounding involved: the vertex and edge results lie on the triangle up to
// the rounding of one fma per coordinate (edge parameters are in [0, 1]
// under correct rounding); the face-region result errs by about
// kappa u |AP|^2 / |edge| for kappa = 1/sin^2 <= 100 (the corner-angle flag),
// unit roundoff u <= 2^-24 and |AP| <= |c - centre| + radius; |c - centre| is
// computed in FP32 from coordinates of magnitude <= max|coordinate|; and the
// computed d2 is within 5u of |p - c|^2.  For |c - centre| <= 50 radius, with
// max|coordinate| <= max|c| + |c - centre|, these become
//   lb >= 0.9449 dc - 1.05 radius - 1e-4 max|c|
//   ub <= 1.0552 dc + 0.05 radius + 1e-4 max|c|,
// evaluated with 0.9438, 1.0501, 1.0563 and 0.0501 for the rounding of the
// sums and of the approximate root (2^-22).  Flagged faces and far ones have
// no bounds.
//
// The faces are taken in short loops, each over this thread's own list, since
// the one loop over all ~30 ring entries that tests a face where it meets it
// runs its test for a few lanes at nearly every entry of the warp:
//   1. of the nearest vertex's ring, the face with the nearest centre is
//      tested;
//   2. the heads of all entries: those with lb above the distance found are
//      dropped, the rest listed;
//   3. of these, the faces that contain an earlier listed vertex are dropped
//      (already met in that vertex's ring with the same inputs);
//   4. the remaining faces (two to four) are tested.
// The smallest squared distance wins, the first entry in the CSR's order on
// ties, as in project_onering's strict '<'.  More than kRingList entries
// listed: project_onering itself.  Bound by the latency of the gathers (the
// warp waits on loads 9 of 16 cycles per instruction at 24 warps per SM).
// Projection kernel on 300k sites and 500k faces, mixed: 114 us with one loop
// over interleaved 64-byte records, 111 with heads apart, 105 so; an FP32
// edge test before the FP64 one (109) and 32 warps (spills; 104) gain nothing.
constexpr int kRingList = 32;
// Entries of step 3 loaded together: one at a time each waits for its own
// load.  Vertex search and projection of 300k sites: 165 us with 1, 158 with 2,
// 157 with 4 (100k sites 76, 74, 76).  Loading the next face of step 4 ahead
// costs spills (160 against 151 us, with the vertex search of grid_knn_box).
constexpr int kRingBatch = 2;
template <int BS> struct RingList { int e[kRingList][BS]; };  // entries, per thread

template <class T, class Q>
__device__ __noinline__ V3<T> project_onering_plain(V3<T> c, const float* __restrict__ V, int nV,
                                                    const int* __restrict__ F, int nF, const int* __restrict__ off,
                                                    const int* __restrict__ fcs, const int* knnv, int kproj) {
  return project_onering<T, Q>(c, V, nV, F, nF, off, fcs, knnv, kproj);
}

__device__ __forceinline__ float approx_root(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// false: more than kRingList faces are left (out is not set)
template <class T, class Q, int BS, int NV>
__device__ __forceinline__ bool project_onering_rec(V3<T> c, const float4* __restrict__ head,
                                                    const float4* __restrict__ body, int nV,
                                                    const int* __restrict__ off, const int (&knnv)[NV],
                                                    RingList<BS>& L, V3<T>& out) {
  const int col = threadIdx.x;
  const float qx = (float)c.x, qy = (float)c.y, qz = (float)c.z;
  const float slack = 1e-4f * fmaxf(fabsf(qx), fmaxf(fabsf(qy), fabsf(qz)));
  int beg[NV], end[NV];
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    const bool valid = (unsigned)knnv[t] < (unsigned)nV;
    beg[t] = valid ? __ldg(off + knnv[t]) : 0;
    end[t] = valid ? __ldg(off + knnv[t] + 1) : 0;
  }
  const V3<Q> cq = cvt3<Q>(c);
  V3<Q> bp = cq;
  Q best = (Q)1e30;
  int best_at = 0;
  auto test = [&](int entry, int at) {
    const float4* w = body + kRingBody * (long)entry;
    const float4 r0 = __ldg(w), r1 = __ldg(w + 1), r2 = __ldg(w + 2);
    if (__float_as_int(r2.y) < 0) return;  // an invalid entry
    const V3<Q> A = {(Q)r0.x, (Q)r0.y, (Q)r0.z};
    const V3<Q> B = {(Q)r0.w, (Q)r1.x, (Q)r1.y};
    const V3<Q> C = {(Q)r1.z, (Q)r1.w, (Q)r2.x};
    const V3<Q> p = closest_point_tri(cq, A, B, C);
    const V3<Q> dd = sub3(p, cq);
    const Q d2 = dot3(dd, dd);
    if (d2 < best || (d2 == best && at < best_at)) { best = d2; bp = p; best_at = at; }
  };
  auto dist = [&](float4 h) {
    const float dx = qx - h.x, dy = qy - h.y, dz = qz - h.z;
    return approx_root(fmaT(dz, dz, fmaT(dy, dy, dx * dx)));
  };
  int first = -1;
  {
    float dmin = INFINITY;
    for (int i = beg[0]; i < end[0]; ++i) {
      const float dc = dist(__ldg(head + i));
      if (dc < dmin) { dmin = dc; first = i; }
    }
  }
  float limit = INFINITY;
  if (first >= 0) {
    test(first, first - end[0]);
    limit = approx_root((float)best) * 1.001f;
  }
  // entries that may hold a nearer point, in the CSR's order; for ties an
  // entry's place is its list index, below 0 in the first ring
  int cnt = 0;
  int ends[NV];  // list length after ring t
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    for (int i0 = beg[t]; i0 < end[t]; i0 += 2) {
      float4 h[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) h[k] = __ldg(head + min(i0 + k, end[t] - 1));
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float dc = dist(h[k]), r = h[k].w;
        if (dc <= 50.f * r && fmaT(0.9438f, dc, -slack) - 1.0501f * r > limit) continue;
        const int i = i0 + k;
        if (i >= end[t] || i == first) continue;
        if (cnt < kRingList) L.e[cnt][col] = i;
        ++cnt;
      }
    }
    ends[t] = cnt;
  }
  if (cnt > kRingList) return false;
  int m = 0, m0 = 0;
  for (int k0 = 0; k0 < cnt; k0 += kRingBatch) {
    int e[kRingBatch];
    float4 ids[kRingBatch];
#pragma unroll
    for (int j = 0; j < kRingBatch; ++j) {
      e[j] = L.e[min(k0 + j, cnt - 1)][col];
      ids[j] = __ldg(body + kRingBody * (long)e[j] + 2);
    }
#pragma unroll
    for (int j = 0; j < kRingBatch; ++j) {
      const int k = k0 + j;
      const int ia = __float_as_int(ids[j].y), ib = __float_as_int(ids[j].z), ic = __float_as_int(ids[j].w);
      bool seen = ia < 0 || k >= cnt;
#pragma unroll
      for (int s = 0; s + 1 < NV; ++s) {
        const int w = knnv[s];
        seen = seen || (k >= ends[s] && (w == ia || w == ib || w == ic));
      }
      if (!seen) L.e[m++][col] = e[j];
      if (k < ends[0]) m0 = m;
    }
  }
  for (int k = 0; k < m; ++k) {
    const int e = L.e[k][col];
    test(e, k < m0 ? e - end[0] : k);
  }
  out = cvt3<T>(bp);
  return true;
}

// project_onering_rec by LANES lanes of a warp (all of the warp takes part):
// the entries of the rings are dealt out to the lanes, each tests the faces
// its entries keep, and the smallest (squared distance, place) of all wins.
// c and knnv are the same in every lane of a group.
template <class T, class Q, int LANES, int NV>
__device__ __forceinline__ V3<T> project_onering_lanes(V3<T> c, const float4* __restrict__ head,
                                                       const float4* __restrict__ body, int nV,
                                                       const int* __restrict__ off, const int (&knnv)[NV]) {
  constexpr unsigned full = 0xffffffffu;
  const int sub = threadIdx.x & (LANES - 1);
  const float qx = (float)c.x, qy = (float)c.y, qz = (float)c.z;
  const float slack = 1e-4f * fmaxf(fabsf(qx), fmaxf(fabsf(qy), fabsf(qz)));
  // entry i of the rings laid end to end is ring t's entry first[t] + i
  int first[NV], end[NV];
  int total = 0;
#pragma unroll
  for (int t = 0; t < NV; ++t) {
    const bool valid = (unsigned)knnv[t] < (unsigned)nV;
    const int b = valid ? __ldg(off + knnv[t]) : 0, e = valid ? __ldg(off + knnv[t] + 1) : 0;
    first[t] = b - total;
    total += e - b;
    end[t] = total;
  }
  auto entry_of = [&](int i, int& t) {
    int f = first[0];
    t = 0;
#pragma unroll
    for (int k = 1; k < NV; ++k)
      if (i >= end[k - 1]) { f = first[k]; t = k; }
    return f + i;
  };
  auto dist = [&](float4 h) {
    const float dx = qx - h.x, dy = qy - h.y, dz = qz - h.z;
    return approx_root(fmaT(dz, dz, fmaT(dy, dy, dx * dx)));
  };
  const V3<Q> cq = cvt3<Q>(c);
  V3<Q> bp = cq;
  Q best = (Q)1e30;
  int best_at = INT_MAX;
  auto test = [&](int entry, int at) {
    const float4* w = body + kRingBody * (long)entry;
    const float4 r0 = __ldg(w), r1 = __ldg(w + 1), r2 = __ldg(w + 2);
    if (__float_as_int(r2.y) < 0) return;  // an invalid entry
    const V3<Q> A = {(Q)r0.x, (Q)r0.y, (Q)r0.z};
    const V3<Q> B = {(Q)r0.w, (Q)r1.x, (Q)r1.y};
    const V3<Q> C = {(Q)r1.z, (Q)r1.w, (Q)r2.x};
    const V3<Q> p = closest_point_tri(cq, A, B, C);
    const V3<Q> dd = sub3(p, cq);
    const Q d2 = dot3(dd, dd);
    if (d2 < best || (d2 == best && at < best_at && best_at != INT_MAX)) { best = d2; bp = p; best_at = at; }
  };
  // the nearest vertex's face with the nearest centre, tested by every lane
  unsigned long long near = ~0ull;
  for (int i = sub; i < end[0]; i += LANES) {
    const unsigned long long k = ((unsigned long long)__float_as_uint(dist(__ldg(head + first[0] + i))) << 32) | (unsigned)i;
    near = k < near ? k : near;
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) {
    const unsigned long long k = __shfl_xor_sync(full, near, o);
    near = k < near ? k : near;
  }
  const int lead = near == ~0ull ? -1 : (int)(unsigned)near;
  float limit = INFINITY;
  if (lead >= 0) {
    test(first[0] + lead, lead);
    limit = approx_root((float)best) * 1.001f;
  }
  for (int i = sub; i < total; i += LANES) {
    int t;
    const int entry = entry_of(i, t);
    const float4 h = __ldg(head + entry);
    const float dc = dist(h);
    if (i == lead || (dc <= 50.f * h.w && fmaT(0.9438f, dc, -slack) - 1.0501f * h.w > limit)) continue;
    const float4 r2 = __ldg(body + kRingBody * (long)entry + 2);
    const int ia = __float_as_int(r2.y), ib = __float_as_int(r2.z), ic = __float_as_int(r2.w);
    bool seen = false;
#pragma unroll
    for (int s = 0; s + 1 < NV; ++s) {
      const int w = knnv[s];
      seen = seen || (s < t && (w == ia || w == ib || w == ic));
    }
    if (!seen) test(entry, i);
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) {
    const Q d = __shfl_xor_sync(full, best, o);
    const int at = __shfl_xor_sync(full, best_at, o);
    const V3<Q> p{__shfl_xor_sync(full, bp.x, o), __shfl_xor_sync(full, bp.y, o), __shfl_xor_sync(full, bp.z, o)};
    if (d < best || (d == best && at < best_at)) { best = d; best_at = at; bp = p; }
  }
  return cvt3<T>(bp);
}

// --------------------------------------------------------------------------
// evaluation primitives (evaluate.cuh:44-104)
// --------------------------------------------------------------------------
// 40-byte BVH node, layout of evaluate.cuh:15-22
struct BVHNode {
  float bmin[3], bmax[3];
  int left, right, triStart, triCount;
};

__device__ __forceinline__ float aabb_d2(V3<float> p, const float* bmin, const float* bmax) {
  float d = 0.f;
  float q[3] = {p.x, p.y, p.z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (q[a] < bmin[a]) { float t = bmin[a] - q[a]; d = fmaT(t, t, d); }
    else if (q[a] > bmax[a]) { float t = q[a] - bmax[a]; d = fmaT(t, t, d); }
  }
  return d;
}

__device__ __forceinline__ float point_tri_d2(V3<float> p, V3<float> a, V3<float> b, V3<float> c) {
  V3<float> ab = sub3(b, a), ac = sub3(c, a), ap = sub3(p, a);
  float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  if (d1 <= 0.f && d2 <= 0.f) return dot3(ap, ap);
  V3<float> bp = sub3(p, b);
  float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
  if (d3 >= 0.f && d4 <= d3) return dot3(bp, bp);
  float vc = fmaT(d1, d4, -(d3 * d2));
  if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
    float v = divT(d1, d1 - d3);
    V3<float> pr{fmaT(ab.x, v, a.x), fmaT(ab.y, v, a.y), fmaT(ab.z, v, a.z)};
    V3<float> d = sub3(p, pr);
    return dot3(d, d);
  }
  V3<float> cp = sub3(p, c);
  float d5 = dot3(ab, cp), d6 = dot3(ac, cp);
  if (d6 >= 0.f && d5 <= d6) return dot3(cp, cp);
  float vb = fmaT(d5, d2, -(d1 * d6));
  if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
    float w = divT(d2, d2 - d6);
    V3<float> pr{fmaT(ac.x, w, a.x), fmaT(ac.y, w, a.y), fmaT(ac.z, w, a.z)};
    V3<float> d = sub3(p, pr);
    return dot3(d, d);
  }
  float va = fmaT(d3, d6, -(d5 * d4));
  if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
    float w = divT(d4 - d3, (d4 - d3) + (d5 - d6));
    V3<float> bc = sub3(c, b);
    V3<float> pr{fmaT(bc.x, w, b.x), fmaT(bc.y, w, b.y), fmaT(bc.z, w, b.z)};
    V3<float> d = sub3(p, pr);
    return dot3(d, d);
  }
  float denom = divT(1.f, (va + vb) + vc);
  float v = vb * denom, w = vc * denom;
  V3<float> pr{a.x + fmaT(ab.x, v, ac.x * w), a.y + fmaT(ab.y, v, ac.y * w), a.z + fmaT(ab.z, v, ac.z * w)};
  V3<float> d = sub3(p, pr);
  return dot3(d, d);
}

// The tree as the traversals read it (k_bvh_pack).  Inner node n has 64
// aligned bytes that hold both children,
//   pair[4n .. 4n+3] = {L.min, L.max.x}, {L.max.yz, R.min.xy},
//                      {R.min.z, R.max}, {left, right, -, -} (ints),
// a child that is a leaf given as ~(its first triangle); the triangles are
// packed in leaf order,
//   tris[3t .. 3t+2] = {A, B.x}, {B.yz, C.xy}, {C.z, last of its leaf, -, -}.
// A step of the descent is four 16-byte loads and a triangle three, where the
// 40-byte nodes took 30 loads of a word and the chain leaf -> face id ->
// corner ids -> corners 13 per triangle.  Hausdorff distance of 900k probes to
// 200k faces: 468 -> 250 us (with the early end in k_hausdorff); projection
// kernel of 50k sites through the BVH: 110 -> 75 us.
struct BvhView {
  const float4* pair;
  const float4* tris;
  float bmin[3], bmax[3];  // the root's box
  int root;                // as a child: 0, or ~0 when the tree is one leaf
};

// Traversal stack: at most one pending sibling per level; the median-split
// tree is at most 2 log2(nF) deep.
constexpr int kBvhStack = 96;

// Near-first traversal of the tree from p: of two children the nearer box is
// entered first, a box only when its FP32 squared distance is below the best
// (limit(), which leaf() may lower).  leaf(t) sees the leaf starting at
// triangle t; false ends the traversal.
template <class Limit, class Leaf>
__device__ __forceinline__ void bvh_walk(const BvhView& v, V3<float> p, int* overflow, Limit limit, Leaf leaf) {
  int stack[kBvhStack];
  float dist[kBvhStack];
  int sp = 0, cur = v.root;
  if (!(aabb_d2(p, v.bmin, v.bmax) < limit())) return;
  while (true) {
    if (cur < 0) {
      if (!leaf(~cur)) return;
    } else {
      const float4* w = v.pair + 4 * (size_t)cur;
      const float4 a = __ldg(w), b = __ldg(w + 1), c = __ldg(w + 2), e = __ldg(w + 3);
      const float lmin[3] = {a.x, a.y, a.z}, lmax[3] = {a.w, b.x, b.y};
      const float rmin[3] = {b.z, b.w, c.x}, rmax[3] = {c.y, c.z, c.w};
      const float dl = aabb_d2(p, lmin, lmax), dr = aabb_d2(p, rmin, rmax);
      const int l = __float_as_int(e.x), r = __float_as_int(e.y);
      if (sp + 2 > kBvhStack) {
        atomicAdd(overflow, 1);
      } else {
        const bool lnear = dl < dr;
        const float dn = lnear ? dl : dr, df = lnear ? dr : dl;
        const int nearer = lnear ? l : r, farther = lnear ? r : l;
        if (df < limit()) { stack[sp] = farther; dist[sp++] = df; }
        if (dn < limit()) { cur = nearer; continue; }
      }
    }
    do {
      if (sp == 0) return;
      --sp;
    } while (!(dist[sp] < limit()));
    cur = stack[sp];
  }
}

// Closest point on the whole mesh through the BVH (projection option; the
// reference projects onto the one-rings of the KPROJ nearest vertices,
// near_project.cuh:149-189).  Near-first traversal; a box is entered only
// when its FP32 squared distance to c is below the best squared distance so
// far, and a face replaces the best only with a strictly smaller squared
// distance, so ties keep the first face met in traversal order.  `best`
// starts at bound2, an upper bound of the answer (the caller's distance to a
// point on the mesh, with margin); if no face beats it the search is rerun
// without the bound.  Q is the barycentric arithmetic type.  The traversal
// order and every comparison are fixed, so a CPU restatement that walks the
// same tree returns the same bits.  A non-finite c is returned unchanged.
template <class T, class Q>
__device__ __forceinline__ V3<T> project_bvh(V3<T> c, const BvhView& bvh, Q bound2, int* overflow) {
  if (!finite3(c)) return c;
  const V3<Q> cq = cvt3<Q>(c);
  const V3<float> cf = cvt3<float>(c);
  V3<Q> bp = cq;
  for (int pass = 0; pass < 2; ++pass) {
    Q best = pass == 0 ? bound2 : (Q)1e30;
    bool found = false;
    bvh_walk(bvh, cf, overflow, [&]() { return best; }, [&](int t) {
      for (bool last = false; !last; ++t) {
        const float4* w = bvh.tris + 3 * (size_t)t;
        const float4 r0 = __ldg(w), r1 = __ldg(w + 1), r2 = __ldg(w + 2);
        last = __float_as_int(r2.y) != 0;
        const V3<Q> A = {(Q)r0.x, (Q)r0.y, (Q)r0.z};
        const V3<Q> B = {(Q)r0.w, (Q)r1.x, (Q)r1.y};
        const V3<Q> C = {(Q)r1.z, (Q)r1.w, (Q)r2.x};
        const V3<Q> p = closest_point_tri(cq, A, B, C);
        const V3<Q> dd = sub3(p, cq);
        const Q d2 = dot3(dd, dd);
        if (d2 < best) { best = d2; bp = p; found = true; }
      }
      return true;
    });
    if (found) break;
  }
  return cvt3<T>(bp);
}

// Upper bound of the squared distance from c to the mesh, given a point s on
// the mesh (up to rounding): (|c - s| (1 + 1e-4) + 1e-5 max|coordinate|)^2.
template <class T>
__device__ __forceinline__ double bvh_bound2(V3<T> c, V3<T> s) {
  const double dx = (double)c.x - (double)s.x, dy = (double)c.y - (double)s.y, dz = (double)c.z - (double)s.z;
  const double m = fmax(fmax(fabs((double)s.x), fabs((double)s.y)), fabs((double)s.z));
  const double d = __dsqrt_rn(__fma_rn(dz, dz, __fma_rn(dy, dy, dx * dx))) * 1.0001 + 1e-5 * m;
  return isfinite(d) ? d * d : 1e30;
}

}  // namespace cvt
