// Stage-API kernels: one kernel (family) per reference stage, operating on
// caller-owned device buffers in the reference's layouts.  They share the
// device routines of the fused engine.
#pragma once
#include "cvt_engine.cuh"
#include "cvt_knn.cuh"

namespace cvt {

// ---------------------------------------------------------------------------
// grid over an arbitrary device point set (geometry chosen on the device)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int f2ord(float v) {
  int b = __float_as_int(v);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float ord2f(int o) {
  int b = o >= 0 ? o : o ^ 0x7fffffff;
  return __int_as_float(b);
}

__global__ void k_bbox_init(int* bb) {
  if (threadIdx.x < 3) { bb[threadIdx.x] = 0x7fffffff; bb[3 + threadIdx.x] = (int)0x80000000; }
}

// Grid-stride blocks with one set of atomics each (a set per warp serialised on
// the six words: 1M points 124 us, now 8).
constexpr int kBboxThreads = 256;
__global__ void __launch_bounds__(kBboxThreads) k_bbox(int n, const float* __restrict__ P, int* bb) {
  __shared__ int sb[6];
  if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? 0x7fffffff : (int)0x80000000;
  __syncthreads();
  int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {(int)0x80000000, (int)0x80000000, (int)0x80000000};
  for (int i = blockIdx.x * kBboxThreads + threadIdx.x; i < n; i += gridDim.x * kBboxThreads) {
    const V3<float> p = ld3(P, i);
    if (!finite3(p)) continue;
    const int o[3] = {f2ord(p.x), f2ord(p.y), f2ord(p.z)};
#pragma unroll
    for (int a = 0; a < 3; ++a) { lo[a] = min(lo[a], o[a]); hi[a] = max(hi[a], o[a]); }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int mn = __reduce_min_sync(0xffffffffu, lo[a]), mx = __reduce_max_sync(0xffffffffu, hi[a]);
    if ((threadIdx.x & 31) == 0) { atomicMin(sb + a, mn); atomicMax(sb + 3 + a, mx); }
  }
  __syncthreads();
  if (threadIdx.x < 3) { if (sb[threadIdx.x] != 0x7fffffff) atomicMin(bb + threadIdx.x, sb[threadIdx.x]); }
  else if (threadIdx.x < 6 && sb[threadIdx.x] != (int)0x80000000) atomicMax(bb + threadIdx.x, sb[threadIdx.x]);
}

// Geometry for ~`per_cell` points per occupied cell on a surface, at most
// max_cells spatial cells (lo, hi: bounds of the finite points, if any).
__device__ inline GridGeom points_geom(bool any, const float* blo, const float* bhi, int n, float per_cell, int max_cells) {
  float lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    lo[a] = any ? blo[a] : 0.f;
    hi[a] = any ? bhi[a] : 1.f;
  }
  float ext[3] = {hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]};
  float emax = fmaxf(fmaxf(ext[0], ext[1]), fmaxf(ext[2], 1e-20f));
  double area = 2.0 * ((double)ext[0] * ext[1] + (double)ext[1] * ext[2] + (double)ext[0] * ext[2]) + 1e-30;
  double h = sqrt(area * per_cell / (double)max(n, 1));
  h = fmax(h, (double)emax / 1024.0);
  GridGeom g;
  for (int it = 0; it < 64; ++it) {
    long long prod = 1;
    for (int a = 0; a < 3; ++a) {
      g.dim[a] = max(1, (int)ceil(((double)ext[a] + 2e-6 * emax) / h));
      prod *= g.dim[a];
    }
    if (prod <= max_cells) break;
    h *= 1.0 + fmax(0.05, cbrt((double)prod / (double)max_cells) - 1.0);
  }
  for (int a = 0; a < 3; ++a) g.lo[a] = lo[a] - 1e-6f * emax;
  g.h = (float)h;
  g.inv_h = (float)(1.0 / h);
  g.cell_base = 0;
  g.ncell = g.dim[0] * g.dim[1] * g.dim[2];
  return g;
}

// Bounds of n points and, by the last block to finish, their grid geometry.
// zero: 8 words that start at zero, so that one memset prepares a whole grid
// build: the bounds as maxima (of the ordered value, and of its complement for
// the lower ones), the ticket in word 6.
__global__ void __launch_bounds__(kBboxThreads) k_bbox_geom(int n, const float* __restrict__ P, unsigned* zero, float per_cell,
                                                            int max_cells, GridGeom* out) {
  __shared__ unsigned sb[6];
  __shared__ bool last;
  if (threadIdx.x < 6) sb[threadIdx.x] = 0u;
  __syncthreads();
  unsigned mx[6] = {0u, 0u, 0u, 0u, 0u, 0u};
  for (int i = blockIdx.x * kBboxThreads + threadIdx.x; i < n; i += gridDim.x * kBboxThreads) {
    const V3<float> p = ld3(P, i);
    if (!finite3(p)) continue;
    const unsigned o[3] = {(unsigned)f2ord(p.x) ^ 0x80000000u, (unsigned)f2ord(p.y) ^ 0x80000000u,
                           (unsigned)f2ord(p.z) ^ 0x80000000u};
#pragma unroll
    for (int a = 0; a < 3; ++a) { mx[a] = max(mx[a], ~o[a]); mx[3 + a] = max(mx[3 + a], o[a]); }
  }
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    const unsigned m = __reduce_max_sync(0xffffffffu, mx[a]);
    if ((threadIdx.x & 31) == 0) atomicMax(sb + a, m);
  }
  __syncthreads();
  if (threadIdx.x < 6) atomicMax(zero + threadIdx.x, sb[threadIdx.x]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(zero + 6, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  float lo[3], hi[3];
  const volatile unsigned* z = zero;
  for (int a = 0; a < 3; ++a) {
    lo[a] = ord2f((int)(~z[a] ^ 0x80000000u));
    hi[a] = ord2f((int)(z[3 + a] ^ 0x80000000u));
  }
  *out = points_geom(z[3] != 0u, lo, hi, n, per_cell, max_cells);
}

// ---------------------------------------------------------------------------
// stage KNN kernels
// ---------------------------------------------------------------------------
template <int KK>
__global__ void __launch_bounds__(128) k_stage_knn_points(const GridGeom* geom, const int* __restrict__ cell_start,
                                                          const Pt4<float>* __restrict__ sorted, int total_cells,
                                                          const uint8_t* frozen, int kk, uint32_t* knn, float* dist) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int n_grid = __ldg(cell_start + total_cells);
  if (t >= n_grid) return;
  const Pt4<float> me = sorted[t];
  const int g = (int)me.id;
  if (frozen && frozen[g]) return;
  TopK<float, KK> top;
  const GridGeom G = *geom;
  grid_knn<float, float, KK>(G, cell_start, sorted, V3<float>{me.x, me.y, me.z}, top, [](uint32_t) { return true; });
#pragma unroll
  for (int k = 0; k < KK; ++k) {
    if (k >= kk) break;
    knn[(size_t)g * kk + k] = KeyOps<float>::idx(top.k[k]);
    if (dist) dist[(size_t)g * kk + k] = KeyOps<float>::dist(top.k[k]);
  }
}

// queries are separate points; out_int != 0 writes int (-1 for missing).  A
// query that has not ended after kQueryRings rings is off the points and is left
// to k_stage_knn_warp with what it found in its row of knn: rest[0] = count,
// then queries.  One thread's ring costs what a warp's does, and a query near
// the points ends with the first: 100k queries, k = 5, to 1M points (us), 1 ring
// / 2 / 4: on the surface 226 / 231 / 229, 3 cells off 322 / 570 / 572, 10 cells
// 795 / 1021 / 2458.
constexpr int kQueryRings = 1;

// Cell ranges that a warp looks up for a query before it scans all points, per
// point.  30k queries, k = 5 (ms), by rings, one thread each, scans alone: 14
// cells off 164k points 0.42, 4.1, 10.5; 40 cells off 1M points 2.7, 36, 65.  A
// query with only empty cells around it pays for the rings and the scan: 60
// cells inside the sphere of 164k points 10.2 together (100 by one thread each).
// 1/2 instead: 60 cells off 20k points 2.7 instead of 1.6.
constexpr float kFarLookups = 0.125f;

template <int KK>
__global__ void __launch_bounds__(128) k_stage_knn_query(const GridGeom* geom, const int* __restrict__ cell_start,
                                                         const Pt4<float>* __restrict__ sorted, const float* __restrict__ Q,
                                                         int nQ, const uint8_t* frozen, int kk, int exclude_self,
                                                         uint32_t* knn, float* dist, int* __restrict__ rest) {
  const int qi = blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= nQ) return;
  if (frozen && frozen[qi]) return;
  TopK<float, KK> top;
  const GridGeom G = *geom;
  const int skip = exclude_self ? qi : -1;
  if (!grid_knn<float, float, KK>(G, cell_start, sorted, ld3(Q, qi), top, [skip](uint32_t id) { return (int)id != skip; },
                                  kQueryRings))
    rest[1 + atomicAdd(rest, 1)] = qi;
#pragma unroll
  for (int k = 0; k < KK; ++k) {
    if (k >= kk) break;
    knn[(size_t)qi * kk + k] = KeyOps<float>::idx(top.k[k]);
    if (dist) dist[(size_t)qi * kk + k] = KeyOps<float>::dist(top.k[k]);
  }
}

// One warp per query (kk <= 32 R): the queries of `rest` ([0] = count), or with
// rest == NULL all n.  Q == NULL: query w is the w-th of the cell-ordered
// points.  Few queries (one thread each would leave most of the chip idle for
// the length of one thread's search) and those that the other kernels leave.
// P != NULL: the queries that k_stage_knn_query left, P the points by index;
// the search goes on where that kernel stopped.
template <int R>
__global__ void __launch_bounds__(128) k_stage_knn_warp(const GridGeom* geom, const int* __restrict__ cell_start,
                                                        const Pt4<float>* __restrict__ sorted, const float* __restrict__ Q,
                                                        int n, const int* __restrict__ rest, const float* __restrict__ P,
                                                        const uint8_t* frozen, int kk, int exclude_self, uint32_t* knn,
                                                        float* dist) {
  const int lane = threadIdx.x & 31;
  const int nw = (int)((gridDim.x * 128u) >> 5);
  const GridGeom G = *geom;
  const int n_pts = __ldg(cell_start + G.cell_base + G.ncell);  // without the non-finite ones
  const int count = rest ? rest[0] : n;
  for (int w = (int)((blockIdx.x * 128u + threadIdx.x) >> 5); w < count; w += nw) {
    const int i = rest ? rest[1 + w] : w;
    V3<float> q;
    int row = i, skip = -1;
    if (Q) {
      q = ld3(Q, i);
      if (exclude_self) skip = i;
    } else {
      const Pt4<float> me = sorted[i];
      q = {me.x, me.y, me.z};
      row = (int)me.id;
    }
    if (frozen && frozen[row]) continue;
    unsigned long long list[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int e = 32 * r + lane;
      list[r] = KeyOps<float>::empty();
      if (P && e < kk) {
        const uint32_t id = knn[(size_t)row * kk + e];
        if (id != 0xffffffffu) list[r] = KeyOps<float>::make(dist2(ld3(P, id), q), id);
      }
    }
    warp_knn_k<float, float, R>(G, cell_start, sorted, n_pts, q, kk, lane, [skip](uint32_t id) { return (int)id != skip; },
                                P ? kQueryRings + 1 : 1, Q ? kFarLookups * (float)n_pts : 0.f, list);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int e = 32 * r + lane;
      if (e < kk) {
        knn[(size_t)row * kk + e] = KeyOps<float>::idx(list[r]);
        if (dist) dist[(size_t)row * kk + e] = KeyOps<float>::dist(list[r]);
      }
    }
  }
}

// Many points with 10 to 40 neighbours each: one warp per 32 consecutive
// points of the cell order (group_knn), rows written by the whole warp.  The
// radius is expected to hold 1.3 kk points at the density of the 27 cells
// around the point (a surface crosses about eleven cells' worth of area
// there).  Left to k_stage_knn_warp: points whose radius holds too few or more
// than 64, and non-finite ones.
__global__ void __launch_bounds__(32, 20) k_stage_knn_group(const GridGeom* geom, const int* __restrict__ cell_start,
                                                        const Pt4<float>* __restrict__ sorted, int n, const uint8_t* frozen,
                                                        int kk, uint32_t* __restrict__ knn, float* __restrict__ dist,
                                                        int* __restrict__ rest) {
  __shared__ GroupPlaces L;
  const int lane = threadIdx.x;
  const GridGeom G = *geom;
  for (int t0 = blockIdx.x * 32; t0 < n; t0 += gridDim.x * 32) {
    const int t = t0 + lane;
    Pt4<float> me{};
    bool in = t < n;
    if (in) {
      me = sorted[t];
      if (frozen && frozen[me.id]) in = false;
    }
    const V3<float> q{me.x, me.y, me.z};
    float thr = 0.f, rad = 0.f;
    if (in && finite3(q)) {
      const int c[3] = {grid_coord(G, q.x, 0), grid_coord(G, q.y, 1), grid_coord(G, q.z, 2)};
      const int x0 = max(c[0] - 1, 0), x1 = min(c[0] + 1, G.dim[0] - 1);
      int near = 0;
      for (int z = max(c[2] - 1, 0); z <= min(c[2] + 1, G.dim[2] - 1); ++z)
        for (int y = max(c[1] - 1, 0); y <= min(c[1] + 1, G.dim[1] - 1); ++y) {
          const int row = G.cell_base + (z * G.dim[1] + y) * G.dim[0];
          near += __ldg(cell_start + row + x1 + 1) - __ldg(cell_start + row + x0);
        }
      thr = (1.3f * 11.f / 3.14159265f) * (float)kk * G.h * G.h / (float)near;
      rad = query_radius(G, q, thr);
    }
    const bool ok = group_knn(G, cell_start, sorted, in, q, thr, rad, kk, L);
    const unsigned left = __ballot_sync(0xffffffffu, in && !ok);
    if (left) {
      int base = 0;
      if (lane == 0) base = atomicAdd(rest, __popc(left));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (in && !ok) rest[1 + base + __popc(left & ((1u << lane) - 1u))] = t;
    }
    for (unsigned rows = __ballot_sync(0xffffffffu, ok); rows; rows &= rows - 1) {
      const int src = __ffs(rows) - 1;
      const V3<float> qs{__shfl_sync(0xffffffffu, q.x, src), __shfl_sync(0xffffffffu, q.y, src),
                         __shfl_sync(0xffffffffu, q.z, src)};
      const size_t row = (size_t)__shfl_sync(0xffffffffu, me.id, src) * kk;
      for (int e = lane; e < kk; e += 32) {
        const Pt4<float> p = sorted[L.at[e][src]];
        knn[row + e] = p.id;
        if (dist) dist[row + e] = dist2(V3<float>{p.x, p.y, p.z}, qs);
      }
    }
    __syncwarp();
  }
}

__global__ void k_stage_drop_self(const uint32_t* __restrict__ in, int n, int kin, int kout, uint32_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t* s = in + (size_t)i * kin;
  uint32_t* d = out + (size_t)i * kout;
  int w = 0;
  for (int t = 0; t < kin && w < kout; ++t) {
    uint32_t j = s[t];
    if ((int)j == i) continue;
    d[w++] = j;
  }
  if (w == 0) {
    for (int k = 0; k < kout; ++k) d[k] = (uint32_t)i;
  } else {
    uint32_t fill = d[w - 1];
    for (; w < kout; ++w) d[w] = fill;
  }
}

__global__ void k_stage_restore_rows(const uint8_t* __restrict__ frozen, const uint32_t* __restrict__ prev,
                                     uint32_t* __restrict__ cur, int n, int k) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !frozen[i]) return;
  for (int a = 0; a < k; ++a) cur[(size_t)i * k + a] = prev[(size_t)i * k + a];
}

// area-weighted vertex normals, summed in face order per vertex
__global__ void k_stage_normals(const float* __restrict__ V, int nV, const int* __restrict__ F,
                                const int* __restrict__ off, const int* __restrict__ fcs, float* __restrict__ N) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nV) return;
  V3<float> acc{0.f, 0.f, 0.f};
  for (int k = off[v]; k < off[v + 1]; ++k) {
    int f = fcs[k];
    V3<float> a = ld3(V, F[3 * f]), b = ld3(V, F[3 * f + 1]), c = ld3(V, F[3 * f + 2]);
    V3<float> fn = cross3(sub3(b, a), sub3(c, a));
    acc = {acc.x + fn.x, acc.y + fn.y, acc.z + fn.z};
  }
  float l2 = dot3(acc, acc);
  if (l2 > 0.f) {
    float inv = divT(1.0f, sqrtT(l2));
    acc = {acc.x * inv, acc.y * inv, acc.z * inv};
  }
  st3(N, v, acc);
}

__global__ void k_stage_frames(const float* __restrict__ N0, const int* __restrict__ knnV, int kproj, int n,
                               float* __restrict__ U, float* __restrict__ Vv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int nn = knnV[(size_t)i * kproj];
  if (nn < 0) { st3(U, i, V3<float>{1, 0, 0}); st3(Vv, i, V3<float>{0, 1, 0}); return; }
  Frame<float> fr = frame_from_normal(ld3(N0, nn));
  st3(U, i, fr.u);
  st3(Vv, i, fr.v);
}

// frames from the PCA normal of each site's listed neighbours (pca_normal),
// started from the normal of the vertex knnV[i * kproj] -- the frame option
// of the engine (frame_mode 1)
__global__ void k_stage_frames_pca(const float* __restrict__ S, int n, const uint32_t* __restrict__ knn, int K,
                                   const float* __restrict__ N0, const int* __restrict__ knnV, int kproj,
                                   float* __restrict__ U, float* __restrict__ Vv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int nn = knnV[(size_t)i * kproj];
  if (nn < 0) { st3(U, i, V3<float>{1, 0, 0}); st3(Vv, i, V3<float>{0, 1, 0}); return; }
  const V3<float> nrm = pca_normal<float>(RowNeighbours<float>{S, knn + (size_t)i * K, (uint32_t)n}, K, ld3(S, i),
                                            ld3(N0, nn));
  Frame<float> fr = frame_from_normal(nrm);
  st3(U, i, fr.u);
  st3(Vv, i, fr.v);
}

// clip + centroid for every site; overflowing polygons go to the fallback
template <int PROF, int BLOCK, int CAP>
__global__ void __launch_bounds__(BLOCK) k_stage_clip(const float* __restrict__ S, const float* __restrict__ U,
                                                      const float* __restrict__ Vv, const uint32_t* __restrict__ knn,
                                                      int n, int K, float R, float* __restrict__ cent, int* nverts,
                                                      int* ovf) {
  using PP = typename PT<PROF>::PP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2<PP>* sm = reinterpret_cast<V2<PP>*>(smem_raw);
  const PolyRef<PP> cur{sm + threadIdx.x, BLOCK};
  const int i = blockIdx.x * BLOCK + threadIdx.x;
  if (i >= n) return;
  V3<float> si = ld3(S, i);
  Frame<float> fr{ld3(U, i), ld3(Vv, i)};
  int np = clip_cell<PROF>(RowNeighbours<float>{S, knn + (size_t)i * K, (uint32_t)n}, si, K, fr, frame_gain(fr.u, fr.v), R, cur,
                           CAP, false);
  if (np < 0) {
    int k = atomicAdd(ovf, 1);
    ovf[1 + k] = i;
    return;
  }
  V2<PP> c2 = poly_centroid<PP>(cur, np, PROF == PROF_MIXED);
  V3<float> c;
  if (!(finiteT(c2.x) && finiteT(c2.y))) c = {NAN, NAN, NAN};
  else {
    float cx = (float)c2.x, cy = (float)c2.y;
    c = {si.x + fmaT(fr.u.x, cx, fr.v.x * cy), si.y + fmaT(fr.u.y, cx, fr.v.y * cy), si.z + fmaT(fr.u.z, cx, fr.v.z * cy)};
  }
  st3(cent, i, c);
  if (nverts) nverts[i] = np;
}

template <int PROF>
__global__ void __launch_bounds__(64) k_stage_clip_fallback(const float* __restrict__ S, const float* __restrict__ U,
                                                            const float* __restrict__ Vv, const uint32_t* __restrict__ knn,
                                                            int n, int K, float R, float* __restrict__ cent, int* nverts,
                                                            const int* ovf) {
  using PP = typename PT<PROF>::PP;
  V2<PP> buf[2][kFallbackCap];
  const int cnt = *ovf;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += gridDim.x * blockDim.x) {
    const int i = ovf[1 + k];
    V3<float> si = ld3(S, i);
    Frame<float> fr{ld3(U, i), ld3(Vv, i)};
    PolyRef<PP> cur{buf[0], 1}, nxt{buf[1], 1};
    int np = clip_cell_full<PROF>(RowNeighbours<float>{S, knn + (size_t)i * K, (uint32_t)n}, si, K, fr, R, cur, nxt, kFallbackCap,
                             false);
    V2<PP> c2 = poly_centroid<PP>(cur, np, PROF == PROF_MIXED);
    V3<float> c;
    if (!(finiteT(c2.x) && finiteT(c2.y))) c = {NAN, NAN, NAN};
    else {
      float cx = (float)c2.x, cy = (float)c2.y;
      c = {si.x + fmaT(fr.u.x, cx, fr.v.x * cy), si.y + fmaT(fr.u.y, cx, fr.v.y * cy), si.z + fmaT(fr.u.z, cx, fr.v.z * cy)};
    }
    st3(cent, i, c);
    if (nverts) nverts[i] = np;
  }
}

template <int PROF>
__global__ void k_stage_project(const float* __restrict__ cent, const float* __restrict__ V, const int* __restrict__ F,
                                const int* __restrict__ off, const int* __restrict__ fcs, const int* __restrict__ knnV,
                                int kproj, int nV, int nF, int nQ, const float* __restrict__ Sold, float* __restrict__ Snew) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nQ) return;
  V3<float> c = ld3(cent, i);
  if (PROF == PROF_MIXED && !finite3(c)) { st3(Snew, i, ld3(Sold, i)); return; }
  int kv[16];
  for (int t = 0; t < kproj && t < 16; ++t) kv[t] = knnV[(size_t)i * kproj + t];
  V3<float> r = (PROF == PROF_REF) ? project_onering<float, float>(c, V, nV, F, nF, off, fcs, kv, min(kproj, 16))
                                   : project_onering<float, double>(c, V, nV, F, nF, off, fcs, kv, min(kproj, 16));
  st3(Snew, i, r);
}

// exact closest point on the mesh through its BVH (project_bvh), the
// projection option of the engine (proj_mode 1); Sold (may be NULL) bounds
// the search and, in MIXED, replaces a non-finite centroid
template <int PROF>
__global__ void k_stage_project_bvh(const float* __restrict__ cent, int nQ, BvhView bvh,
                                    const float* __restrict__ Sold, float* __restrict__ Snew, int* ovf) {
  using Q = typename PT<PROF>::Q;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nQ) return;
  V3<float> c = ld3(cent, i);
  if (PROF == PROF_MIXED && !finite3(c)) { st3(Snew, i, ld3(Sold, i)); return; }
  const Q bound2 = Sold ? (Q)bvh_bound2(c, ld3(Sold, i)) : (Q)1e30;
  st3(Snew, i, project_bvh<float, Q>(c, bvh, bound2, ovf));
}

struct FreezeTable { float thr2[6]; int need[6]; };

__global__ void k_stage_freeze(const float* __restrict__ S, const float* __restrict__ Snew,
                               const uint32_t* __restrict__ knn, const uint32_t* __restrict__ prev, int n, int K,
                               int has_prev, const uint8_t* __restrict__ tier, FreezeTable tab, uint8_t* streak,
                               uint8_t* cand, uint8_t* frozen, int* counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int same = 0, low = 0, both = 0, newly = 0;
  if (i < n) {
    if (!has_prev) {
      streak[i] = 0;
      cand[i] = 0;
    } else {
      int t = tier ? min((int)tier[i], 5) : 0;
      bool sm = true;
      for (int j = 0; j < K; ++j)
        if (knn[(size_t)i * K + j] != prev[(size_t)i * K + j]) { sm = false; break; }
      bool lw = dist2(ld3(Snew, i), ld3(S, i)) <= tab.thr2[t];
      bool bt = sm && lw;
      int s = streak[i];
      s = bt ? (s < 255 ? s + 1 : s) : 0;
      streak[i] = (uint8_t)s;
      uint8_t c = (s >= tab.need[t]) ? 1 : 0;
      cand[i] = c;
      same = sm; low = lw; both = bt;
      if (c && !frozen[i]) { frozen[i] = 1; newly = 1; }
    }
  }
  const unsigned full = 0xffffffffu;
  int a = __popc(__ballot_sync(full, same)), b = __popc(__ballot_sync(full, low));
  int c = __popc(__ballot_sync(full, both)), d = __popc(__ballot_sync(full, newly));
  if ((threadIdx.x & 31) == 0) {
    if (a) atomicAdd(counts + 0, a);
    if (b) atomicAdd(counts + 1, b);
    if (c) atomicAdd(counts + 2, c);
    if (d) atomicAdd(counts + 3, d);
  }
}

__global__ void k_stage_count_frozen(const uint8_t* __restrict__ frozen, int n, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int v = (i < n && frozen[i]) ? 1 : 0;
  int c = __popc(__ballot_sync(0xffffffffu, v));
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

__global__ void k_stage_tiers(int mode, int n, int K, const float* __restrict__ sn, const uint32_t* __restrict__ knn,
                              uint8_t* __restrict__ tier) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  auto normal = [&](int j, float out[3]) { out[0] = sn[3 * j]; out[1] = sn[3 * j + 1]; out[2] = sn[3 * j + 2]; };
  auto row = [&](int t) {
    const int j = (int)knn[(size_t)i * K + t];
    return j < n ? j : -1;
  };
  tier[i] = (uint8_t)tier_of(mode, i, K, row, normal);
}

}  // namespace cvt
