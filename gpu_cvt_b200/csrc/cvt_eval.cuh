// Evaluation: BVH traversal over the reference surface and the one-sided Hausdorff
// distance of a candidate mesh (evaluate.cuh:15-383), plus the dual-triangle
// extraction that produces the candidate mesh from the sites
// (near_project.cuh:201-352, buildmesh.cuh:11-241, main.cu:928-974).
#pragma once
#include <algorithm>
#include <vector>
#include "cvt_engine.cuh"

namespace cvt {

// The tree is the reference's (bounds from the triangle boxes, leaf <= 8
// triangles, otherwise the centroid-sorted list split at its middle, nodes in
// pre-order, evaluate.cuh:114-201); it is built on the device, cvt_ingest.cuh.

// Closest squared distance of p to the surface (the traversal order only
// changes the order, not the minimum), or any value <= floor2() once it is
// known not to be above that (floor2 is looked at once per leaf).
template <class Floor>
__device__ __forceinline__ float bvh_closest_d2(V3<float> p, const BvhView& bvh, int* overflow, Floor floor2) {
  float best = 1e30f;
  bvh_walk(bvh, p, overflow, [&]() { return best; }, [&](int t) {
    const float fl = floor2();
    for (bool last = false; !last; ++t) {
      const float4* w = bvh.tris + 3 * (size_t)t;
      const float4 r0 = __ldg(w), r1 = __ldg(w + 1), r2 = __ldg(w + 2);
      last = __float_as_int(r2.y) != 0;
      const float d2 = point_tri_d2(p, {r0.x, r0.y, r0.z}, {r0.w, r1.x, r1.y}, {r1.z, r1.w, r2.x});
      if (d2 < best) {
        best = d2;
        if (best <= fl) return false;
      }
    }
    return true;
  });
  return best;
}

// probe k of the candidate mesh: vertices, then per face the centroid and
// the three edge midpoints (evaluate.cuh:253-283)
__device__ __forceinline__ V3<float> probe_point(const float* __restrict__ V, int nV, const int* __restrict__ F, long k) {
  if (k < nV) return ld3(V, k);
  long f = (k - nV) >> 2;
  int w = (int)((k - nV) & 3);
  V3<float> a = ld3(V, F[3 * f]), b = ld3(V, F[3 * f + 1]), c = ld3(V, F[3 * f + 2]);
  const float third = 1.0f / 3.0f;
  if (w == 0) return {(a.x + (b.x + c.x)) * third, (a.y + (b.y + c.y)) * third, (a.z + (b.z + c.z)) * third};
  if (w == 1) return {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
  if (w == 2) return {(b.x + c.x) * 0.5f, (b.y + c.y) * 0.5f, (b.z + c.z) * 0.5f};
  return {(c.x + a.x) * 0.5f, (c.y + a.y) * 0.5f, (c.z + a.z) * 0.5f};
}

// max over probes of the closest squared distance, reduced in-kernel:
// warp max, then one atomicMax on the float bits (non-negative floats
// order as unsigned ints) -- replaces the CUB max of evaluate.cuh:335-343.
// A probe whose closest distance so far is not above the maximum of the
// probes already done cannot raise it and stops there, which ends most of
// them at their first leaf; the maximum is the same.
__global__ void __launch_bounds__(128) k_hausdorff(const float* __restrict__ Vc, int nVc, const int* __restrict__ Fc,
                                                   long nP, BvhView bvh, unsigned* out_bits, int* overflow) {
  long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  float d = 0.f;
  if (k < nP)
    d = bvh_closest_d2(probe_point(Vc, nVc, Fc, k), bvh, overflow,
                       [&]() { return __uint_as_float(*(volatile unsigned*)out_bits); });
  unsigned b = __float_as_uint(d);
  b = __reduce_max_sync(0xffffffffu, b);
  if ((threadIdx.x & 31) == 0 && b > *(volatile unsigned*)out_bits) atomicMax(out_bits, b);
}

// ---------------------------------------------------------------------------
// dual-triangle extraction
// ---------------------------------------------------------------------------
// Neighbour lists of k_face_keys: get(i, t) is entry t of site i's list (an
// index into the sites, or out of range), label(i) the index that a site has
// in the faces.
struct FaceRows {  // row-major lists
  const uint32_t* knn;
  int K;
  __device__ __forceinline__ int get(int i, int t) const { return (int)knn[(size_t)i * K + t]; }
  __device__ __forceinline__ int label(int i) const { return i; }
};
struct FaceLists {  // an engine segment's lists (from its first site on)
  const uint32_t* list;
  const int* labels;
  size_t site, entry;  // EngineArgs::list_site, list_entry
  uint32_t base;
  __device__ __forceinline__ int get(int i, int t) const {
    const uint32_t j = list[i * site + t * entry];
    return j == 0xffffffffu ? -1 : (int)(j - base);
  }
  __device__ __forceinline__ int label(int i) const { return labels[i]; }
};

// Labelled clip (near_project.cuh:201-244) + active-bisector pairs
// (near_project.cuh:318-351) + key emission (buildmesh.cuh:170-201) per site.

__device__ __forceinline__ void face_emit(int x, int y, int z, unsigned long long* keys, int* key_count, int max_keys) {
  int tmp;
  if (x > y) { tmp = x; x = y; y = tmp; }
  if (y > z) { tmp = y; y = z; z = tmp; }
  if (x > y) { tmp = x; x = y; y = tmp; }
  const int pos = atomicAdd(key_count, 1);
  if (pos < max_keys)
    keys[pos] = (unsigned long long)(uint32_t)x | ((unsigned long long)(uint32_t)y << 21) |
                ((unsigned long long)(uint32_t)z << 42);
}

// One site per thread, the polygon in shared memory (kFaceCap vertices), cut
// in place by outside masks as clip_cell does; sites that need more vertices
// or whose outside vertices are not one run go to `over` (k_face_keys_over).
// The clip's labels only name the edges, which the faces do not use: a face
// joins the site and the two listed neighbours whose bisectors pass nearest a
// vertex, both within tol_active; neighbours beyond it cannot be among them,
// so one pass over the neighbours finds both for every vertex.  100k sites,
// K = 24: 148 us with 256-vertex buffers in local memory and all neighbours'
// bisectors recomputed for every vertex, now 110.
constexpr int kFaceThreads = 64;
constexpr int kFaceCap = 16;

template <class NB>
__global__ void __launch_bounds__(kFaceThreads) k_face_keys(const float* __restrict__ S, const float* __restrict__ U,
                                                            const float* __restrict__ Vv, NB nb, int n, int K, float R2,
                                                            float eps_clip, float tol_active, unsigned long long* keys,
                                                            int* key_count, int max_keys, int* __restrict__ over) {
  __shared__ float2 P[kFaceCap][kFaceThreads];
  __shared__ float2 near_d[kFaceCap][kFaceThreads];  // the two smallest |f| within tol_active
  __shared__ int2 near_j[kFaceCap][kFaceThreads];
  const int c = threadIdx.x, i = blockIdx.x * kFaceThreads + threadIdx.x;
  if (i >= n) return;
  const V3<float> si = ld3(S, i), ui = ld3(U, i), vi = ld3(Vv, i);
  P[0][c] = make_float2(-R2, -R2); P[1][c] = make_float2(R2, -R2); P[2][c] = make_float2(R2, R2); P[3][c] = make_float2(-R2, R2);
  int na = 4;
  const float gain = frame_gain(ui, vi);
  float r2 = 2.f * R2 * R2 * 1.0001f;
  for (int t = 0; t < K; ++t) {
    if (na <= 0) continue;
    const int j = nb.get(i, t);
    if ((unsigned)j >= (unsigned)n || j == i) continue;
    const V3<float> d = sub3(ld3(S, j), si);
    const float dd = dot3(d, d);
    if (dd > 4.01f * gain * r2 && dd > 2e-18f && dd < 1e30f) continue;  // cannot cut (clip_cell)
    const float a = dot3(d, ui), b = dot3(d, vi), cc = 0.5f * dd;
    auto f = [&](float2 p) { return fmaT(a, p.x, fmaT(b, p.y, -cc)); };
    unsigned out = 0u;
    float rin = 0.f;
    for (int k = 0; k < na; ++k) {
      const float2 p = P[k][c];
      if (f(p) <= eps_clip) rin = fmaxf(rin, fmaT(p.y, p.y, p.x * p.x)); else out |= 1u << k;
    }
    if (out == 0u) continue;
    const unsigned all = 0xffffffffu >> (32 - na);
    if (out == all) { na = 0; continue; }
    const unsigned starts = out & ~((out << 1) | (out >> (na - 1)));
    const int len = __popc(out), p0 = __ffs(starts) - 1;
    if ((starts & (starts - 1)) || na - len + 2 > kFaceCap) { na = -1; continue; }
    const int q = p0 + len - 1 >= na ? p0 + len - 1 - na : p0 + len - 1;
    const int ip = p0 == 0 ? na - 1 : p0 - 1, iq = q + 1 == na ? 0 : q + 1;
    auto isect = [&](float2 s, float2 e) {
      const float fs = f(s), fe = f(e);
      const float tt = divT(fs, (fs - fe) + 1e-30f);
      return make_float2(fmaT(tt, e.x - s.x, s.x), fmaT(tt, e.y - s.y, s.y));
    };
    const float2 enter = isect(P[ip][c], P[p0][c]), leave = isect(P[q][c], P[iq][c]);
    int lo, hi, shift, at_enter, at_leave;
    if (p0 <= q && q + 1 < na) { lo = q + 1; hi = na; shift = 2 - len; at_enter = p0; at_leave = p0 + 1; }
    else { lo = iq; hi = p0; shift = 1 - iq; at_enter = na - len + 1; at_leave = 0; }
    if (shift > 0) { for (int k = hi - 1; k >= lo; --k) P[k + shift][c] = P[k][c]; }
    else if (shift < 0) { for (int k = lo; k < hi; ++k) P[k + shift][c] = P[k][c]; }
    P[at_enter][c] = enter;
    P[at_leave][c] = leave;
    na += 2 - len;
    const float re = fmaT(enter.y, enter.y, enter.x * enter.x), rl = fmaT(leave.y, leave.y, leave.x * leave.x);
    r2 = fmaxf(rin, fmaxf(re, rl)) * 1.000001f;
    if (!(re < INFINITY) || !(rl < INFINITY)) na = -1;
  }
  if (na < 0) { over[1 + atomicAdd(over, 1)] = i; return; }
  if (na < 3) return;
  for (int k = 0; k < na; ++k) { near_d[k][c] = make_float2(1e30f, 1e30f); near_j[k][c] = make_int2(-1, -1); }
  for (int t = 0; t < K; ++t) {
    const int j = nb.get(i, t);
    if ((unsigned)j >= (unsigned)n || j == i) continue;
    const V3<float> d = sub3(ld3(S, j), si);
    const float a = dot3(d, ui), b = dot3(d, vi), cc = 0.5f * dot3(d, d);
    for (int k = 0; k < na; ++k) {
      const float2 p = P[k][c];
      const float s = fabsf(fmaT(a, p.x, fmaT(b, p.y, -cc)));
      if (!(s <= tol_active)) continue;
      float2 nd = near_d[k][c];
      int2 nj = near_j[k][c];
      if (s < nd.x) { nd.y = nd.x; nj.y = nj.x; nd.x = s; nj.x = j; }
      else if (s < nd.y) { nd.y = s; nj.y = j; }
      near_d[k][c] = nd; near_j[k][c] = nj;
    }
  }
  for (int k = 0; k < na; ++k) {
    const int2 nj = near_j[k][c];
    if (nj.x >= 0 && nj.y >= 0 && nj.x != nj.y)
      face_emit(nb.label(i), nb.label(nj.x), nb.label(nj.y), keys, key_count, max_keys);
  }
}

// The sites that k_face_keys gave back, with the reference's two buffers of
// kFaceMaxPoly vertices (MAX_POLY, main.cu:393) in local memory.
constexpr int kFaceMaxPoly = 256;

template <class NB>
__global__ void __launch_bounds__(64) k_face_keys_over(const float* __restrict__ S, const float* __restrict__ U,
                                                       const float* __restrict__ Vv, NB nb, int n, int K, float R2,
                                                       float eps_clip, float tol_active, unsigned long long* keys,
                                                       int* key_count, int max_keys, const int* __restrict__ over) {
  float2 bufA[kFaceMaxPoly], bufB[kFaceMaxPoly];
  const int n_over = over[0];
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n_over; w += gridDim.x * blockDim.x) {
    const int i = over[1 + w];
    float2* cp = bufA; float2* np = bufB;
    int na = 4;
    cp[0] = make_float2(-R2, -R2); cp[1] = make_float2(R2, -R2); cp[2] = make_float2(R2, R2); cp[3] = make_float2(-R2, R2);
    const V3<float> si = ld3(S, i), ui = ld3(U, i), vi = ld3(Vv, i);
    for (int t = 0; t < K && na > 0; ++t) {
      const int j = nb.get(i, t);
      if ((unsigned)j >= (unsigned)n || j == i) continue;
      const V3<float> d = sub3(ld3(S, j), si);
      const float a = dot3(d, ui), b = dot3(d, vi), c = 0.5f * dot3(d, d);
      int m = 0;
      float2 s = cp[na - 1];
      float fs = fmaT(a, s.x, fmaT(b, s.y, -c));
      for (int k = 0; k < na; ++k) {
        const float2 e = cp[k];
        const float fe = fmaT(a, e.x, fmaT(b, e.y, -c));
        const bool ins_e = fe <= eps_clip, ins_s = fs <= eps_clip;
        if (ins_e != ins_s && m < kFaceMaxPoly) {
          const float tt = divT(fs, (fs - fe) + 1e-30f);
          np[m++] = make_float2(fmaT(tt, e.x - s.x, s.x), fmaT(tt, e.y - s.y, s.y));
        }
        if (ins_e && m < kFaceMaxPoly) np[m++] = e;
        s = e; fs = fe;
      }
      na = m;
      float2* tp = cp; cp = np; np = tp;
    }
    if (na < 3) continue;
    for (int k = 0; k < na; ++k) {
      const float2 p = cp[k];
      float b1 = 1e30f, b2 = 1e30f;
      int j1 = -1, j2 = -1;
      for (int t = 0; t < K; ++t) {
        const int j = nb.get(i, t);
        if ((unsigned)j >= (unsigned)n || j == i) continue;
        const V3<float> d = sub3(ld3(S, j), si);
        const float a = dot3(d, ui), b = dot3(d, vi), c = 0.5f * dot3(d, d);
        const float s = fabsf(fmaT(a, p.x, fmaT(b, p.y, -c)));
        if (s < b1) { b2 = b1; j2 = j1; b1 = s; j1 = j; }
        else if (s < b2) { b2 = s; j2 = j; }
      }
      if (j1 >= 0 && j2 >= 0 && j1 != j2 && b1 <= tol_active && b2 <= tol_active)
        face_emit(nb.label(i), nb.label(j1), nb.label(j2), keys, key_count, max_keys);
    }
  }
}

}  // namespace cvt

namespace cvt {

// decode the sorted unique keys (buildmesh.cuh:99-109) and drop degenerate
// triangles (buildmesh.cuh:225-241, eps 1e-6); flags[k] = keep
__global__ void k_face_decode(const unsigned long long* __restrict__ keys, int nk, const float* __restrict__ S, int n,
                              float eps, int* __restrict__ tri, int* __restrict__ keep) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nk) return;
  unsigned long long key = keys[k];
  int a = (int)(key & 0x1FFFFFull), b = (int)((key >> 21) & 0x1FFFFFull), c = (int)((key >> 42) & 0x1FFFFFull);
  bool deg = (a == b || b == c || a == c) || a >= n || b >= n || c >= n;
  if (!deg) {
    V3<float> A = ld3(S, a), B = ld3(S, b), C = ld3(S, c);
    V3<float> e0 = sub3(B, A), e1 = sub3(C, B), e2 = sub3(A, C);
    float l0 = sqrtT(dot3(e0, e0)), l1 = sqrtT(dot3(e1, e1)), l2 = sqrtT(dot3(e2, e2));
    V3<float> cr = cross3(sub3(B, A), sub3(C, A));
    float ar = sqrtT(dot3(cr, cr));
    deg = !(l0 > eps && l1 > eps && l2 > eps && ar > eps);
  }
  tri[3 * k] = a; tri[3 * k + 1] = b; tri[3 * k + 2] = c;
  keep[k] = deg ? 0 : 1;
}

__global__ void k_face_compact(const int* __restrict__ tri, const int* __restrict__ keep, const int* __restrict__ pos,
                               int nk, int* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nk || !keep[k]) return;
  int p = pos[k];
  out[3 * p] = tri[3 * k]; out[3 * p + 1] = tri[3 * k + 1]; out[3 * p + 2] = tri[3 * k + 2];
}

// quality metrics (evaluate.cuh:388-462) as a device reduction: acc[0] Qsum,
// acc[1] min-angle sum, acc[2] #angles < 30, acc[3] #angles > 90 (doubles);
// mins[0] Qmin bits, mins[1] theta_min bits (non-negative floats as uint)
// Grid-stride blocks, one set of atomics per block (per warp: 43 us for 200k
// faces, now 8).
constexpr int kQualityThreads = 256;
__global__ void __launch_bounds__(kQualityThreads) k_quality(const float* __restrict__ V, const int* __restrict__ F, int nF,
                                                             double* acc, unsigned* mins) {
  __shared__ double sacc[4];
  __shared__ unsigned smin[2];
  if (threadIdx.x < 4) sacc[threadIdx.x] = 0.0;
  if (threadIdx.x < 2) smin[threadIdx.x] = 0x7f7f7f7fu;
  __syncthreads();
  double q = 0.0, th = 0.0, lt = 0.0, gt = 0.0;
  float qmin = 3.0e38f, tmin = 3.0e38f;
  for (int f = blockIdx.x * kQualityThreads + threadIdx.x; f < nF; f += gridDim.x * kQualityThreads) {
    V3<float> a = ld3(V, F[3 * f]), b = ld3(V, F[3 * f + 1]), c = ld3(V, F[3 * f + 2]);
    V3<float> ab = sub3(b, a), ac = sub3(c, a), ba = sub3(a, b), bc = sub3(c, b), ca = sub3(a, c), cb = sub3(b, c);
    auto ang = [](V3<float> u, V3<float> v) {
      float du = sqrtT(dot3(u, u)), dv = sqrtT(dot3(v, v));
      float den = fmaxf(du * dv, 1e-30f);
      float cs = divT(dot3(u, v), den);
      cs = fminf(1.f, fmaxf(-1.f, cs));
      return acosf(cs) * (180.0f / 3.14159265358979323846f);
    };
    float A = ang(ab, ac), B = ang(ba, bc), Cc = ang(ca, cb);
    const float tm = fminf(A, fminf(B, Cc));
    tmin = fminf(tmin, tm);
    th += tm;
    lt += (A < 30.f) + (B < 30.f) + (Cc < 30.f);
    gt += (A > 90.f) + (B > 90.f) + (Cc > 90.f);
    float l0 = sqrtT(dot3(ab, ab)), l1 = sqrtT(dot3(bc, bc)), l2 = sqrtT(dot3(ca, ca));
    V3<float> cr = cross3(ab, ac);
    float area = 0.5f * sqrtT(dot3(cr, cr));
    float s = 0.5f * ((l0 + l1) + l2);
    float e = fmaxf(l0, fmaxf(l1, l2));
    float den = fmaxf(s * e, 1e-30f);
    float qq = divT(6.0f, sqrtT(3.0f)) * divT(area, den);
    qmin = fminf(qmin, qq);
    q += qq;
  }
  for (int o = 16; o; o >>= 1) {
    q += __shfl_xor_sync(0xffffffffu, q, o);
    th += __shfl_xor_sync(0xffffffffu, th, o);
    lt += __shfl_xor_sync(0xffffffffu, lt, o);
    gt += __shfl_xor_sync(0xffffffffu, gt, o);
    qmin = fminf(qmin, __shfl_xor_sync(0xffffffffu, qmin, o));
    tmin = fminf(tmin, __shfl_xor_sync(0xffffffffu, tmin, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(sacc + 0, q); atomicAdd(sacc + 1, th); atomicAdd(sacc + 2, lt); atomicAdd(sacc + 3, gt);
    atomicMin(smin + 0, __float_as_uint(qmin));
    atomicMin(smin + 1, __float_as_uint(tmin));
  }
  __syncthreads();
  if (threadIdx.x < 4) atomicAdd(acc + threadIdx.x, sacc[threadIdx.x]);
  if (threadIdx.x < 2) atomicMin(mins + threadIdx.x, smin[threadIdx.x]);
}

}  // namespace cvt
