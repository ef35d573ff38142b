// Uniform-grid spatial hash and exact K-nearest-neighbour search.
//
// Replaces the reference's random-hub index (bitonic-hubs-grid.cuh:1142-1656,
// rebuilt with ~20 cudaMalloc per call, host shuffles and H x H bound
// matrices) with a per-segment uniform grid rebuilt by a counting sort every
// iteration.  The answer is the exact K nearest points in (squared distance,
// index) order; the search widens ring by ring until the K-th candidate is
// provably closer than every unvisited cell, so the result does not depend
// on the cell size (only the time does).
#pragma once
#include "cvt_math.cuh"

namespace cvt {

// Grid over one segment's points.  Cells [cell_base, cell_base + ncell) are
// spatial (x fastest); cell_base + ncell is the bucket of non-finite points,
// which is never searched.
struct GridGeom {
  float lo[3];
  float h, inv_h;
  int dim[3];
  int cell_base;
  int ncell;
};

// Cell-ordered copy of a point: coordinates plus the point's global index.
template <class T> struct alignas(16) Pt4 { T x, y, z; uint32_t id; };

// position of point i (one 16-byte load; FP64: two)
template <class T> __device__ __forceinline__ V3<T> ldp(const Pt4<T>* __restrict__ P, uint32_t i) {
  const Pt4<T> p = P[i];
  return {p.x, p.y, p.z};
}

template <class T>
__device__ __forceinline__ int grid_coord(const GridGeom& g, T v, int a) {
  float f = floorf(((float)v - g.lo[a]) * g.inv_h);
  int c = (f >= 0.f) ? (f < (float)g.dim[a] ? (int)f : g.dim[a] - 1) : 0;
  return c;
}

template <class T>
__device__ __forceinline__ int grid_cell(const GridGeom& g, V3<T> p) {
  if (!finite3(p)) return g.cell_base + g.ncell;
  int cx = grid_coord(g, p.x, 0), cy = grid_coord(g, p.y, 1), cz = grid_coord(g, p.z, 2);
  return g.cell_base + (cz * g.dim[1] + cy) * g.dim[0] + cx;
}

// ---------------------------------------------------------------------------
// top-K with (distance, index) keys
// ---------------------------------------------------------------------------
template <class T> struct KeyOps;

// float: the key is (float bits << 32 | index); non-negative floats order as
// their bit patterns, so one 64-bit compare orders by distance then index.
template <> struct KeyOps<float> {
  using Key = unsigned long long;
  static __device__ __forceinline__ Key make(float d, uint32_t i) {
    return ((Key)__float_as_uint(d) << 32) | (Key)i;
  }
  static __device__ __forceinline__ Key empty() { return ~0ull; }
  static __device__ __forceinline__ bool less(Key a, Key b) { return a < b; }
  static __device__ __forceinline__ Key kmin(Key a, Key b) { return a < b ? a : b; }
  static __device__ __forceinline__ Key kmax(Key a, Key b) { return a < b ? b : a; }
  static __device__ __forceinline__ uint32_t idx(Key k) { return (uint32_t)(k & 0xffffffffull); }
  static __device__ __forceinline__ float dist(Key k) {
    return k == ~0ull ? __int_as_float(0x7f800000) : __uint_as_float((uint32_t)(k >> 32));
  }
  static __device__ __forceinline__ bool is_empty(Key k) { return k == ~0ull; }
};

struct DKey { double d; uint32_t i; };
template <> struct KeyOps<double> {
  using Key = DKey;
  static __device__ __forceinline__ Key make(double d, uint32_t i) { return {d, i}; }
  static __device__ __forceinline__ Key empty() { return {__longlong_as_double(0x7ff0000000000000ll), 0xffffffffu}; }
  static __device__ __forceinline__ bool less(Key a, Key b) { return a.d < b.d || (a.d == b.d && a.i < b.i); }
  static __device__ __forceinline__ Key kmin(Key a, Key b) { return less(a, b) ? a : b; }
  static __device__ __forceinline__ Key kmax(Key a, Key b) { return less(a, b) ? b : a; }
  static __device__ __forceinline__ uint32_t idx(Key k) { return k.i; }
  static __device__ __forceinline__ double dist(Key k) { return k.d; }
  static __device__ __forceinline__ bool is_empty(Key k) { return k.i == 0xffffffffu && isinf(k.d); }
};

// Sorted register list; insertion keeps the KK smallest keys.  Branch-free
// update new[j] = max(old[j-1], min(old[j], x)) keeps the list in registers.
template <class T, int KK> struct TopK {
  using O = KeyOps<T>;
  typename O::Key k[KK];
  __device__ __forceinline__ TopK() {
#pragma unroll
    for (int j = 0; j < KK; ++j) k[j] = O::empty();
  }
  __device__ __forceinline__ T worst_d() const { return O::dist(k[KK - 1]); }
  __device__ __forceinline__ bool full() const { return !O::is_empty(k[KK - 1]); }
  __device__ __forceinline__ void insert(typename O::Key x) {
    if (!O::less(x, k[KK - 1])) return;
#pragma unroll
    for (int j = KK - 1; j > 0; --j) k[j] = O::kmax(k[j - 1], O::kmin(k[j], x));
    k[0] = O::kmin(k[0], x);
  }
};

// Exact KK-nearest search of q among the points of one grid.  accept(id)
// filters candidates (used for the vertex-index exclusion quirk).
// With rlim > 0 the search gives up (returns false, top incomplete) when it
// has not finished after rlim rings: a query far from every point would
// otherwise visit the whole grid, one cell at a time.
template <class T, class PT, int KK, class Accept>
__device__ __forceinline__ bool grid_knn(const GridGeom& g, const int* __restrict__ cell_start,
                                         const Pt4<PT>* __restrict__ pts, V3<T> q, TopK<T, KK>& top,
                                         Accept accept, int rlim = 0) {
  if (!finite3(q)) return true;
  const int cx = grid_coord(g, q.x, 0), cy = grid_coord(g, q.y, 1), cz = grid_coord(g, q.z, 2);
  const int rmax = max(g.dim[0], max(g.dim[1], g.dim[2]));
  const float slack = 1e-3f * g.h;
  const float qf[3] = {(float)q.x, (float)q.y, (float)q.z};
  const int c[3] = {cx, cy, cz};
  auto scan_range = [&](int b, int e) {
    for (int k = b; k < e; ++k) {
      Pt4<PT> p = pts[k];
      if (!accept(p.id)) continue;
      T d = dist2(V3<T>{(T)p.x, (T)p.y, (T)p.z}, q);
      if (d <= top.worst_d()) top.insert(KeyOps<T>::make(d, p.id));
    }
  };
  for (int r = 1; r <= rmax; ++r) {
    const int z0 = max(cz - r, 0), z1 = min(cz + r, g.dim[2] - 1);
    const int y0 = max(cy - r, 0), y1 = min(cy + r, g.dim[1] - 1);
    const int x0 = max(cx - r, 0), x1 = min(cx + r, g.dim[0] - 1);
    for (int z = z0; z <= z1; ++z) {
      for (int y = y0; y <= y1; ++y) {
        const int row = g.cell_base + (z * g.dim[1] + y) * g.dim[0];
        const bool full_row = (r == 1) || abs(z - cz) == r || abs(y - cy) == r;
        if (full_row) {
          scan_range(__ldg(cell_start + row + x0), __ldg(cell_start + row + x1 + 1));
        } else {
          if (cx - r >= 0) scan_range(__ldg(cell_start + row + cx - r), __ldg(cell_start + row + cx - r + 1));
          if (cx + r < g.dim[0]) scan_range(__ldg(cell_start + row + cx + r), __ldg(cell_start + row + cx + r + 1));
        }
      }
    }
    // lower bound on the distance to any point outside the visited block
    float m = __int_as_float(0x7f800000);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (c[a] - r > 0) m = fminf(m, qf[a] - (g.lo[a] + (float)(c[a] - r) * g.h));
      if (c[a] + r < g.dim[a] - 1) m = fminf(m, (g.lo[a] + (float)(c[a] + r + 1) * g.h) - qf[a]);
    }
    if (isinf(m)) break;
    m -= slack;
    if (top.full() && m > 0.f && (double)top.worst_d() < (double)m * (double)m) break;
    if (r == rlim) return false;
  }
  return true;
}

// The KK nearest points of q from one box query (one thread): every
// accepted point of the cells in q +- rad with squared distance <= thr is
// offered to top.  When top fills, it holds the KK nearest in (squared
// distance, index) order, the keys grid_knn returns: a point left out is
// farther than thr, so farther than every key kept.  rad must cover
// sqrt(thr) with margin (cell coordinates are monotone in the position).
// Returns false, top partly filled, when fewer than KK points pass or the
// box spans more than max_cells cells; the caller then resets top and runs
// grid_knn.
// One loop over the points of all rows, two a step, with the next row's range
// on its way: a loop per row made a warp take the longest row of its lanes
// every time (12 of 32 threads active) and wait for each row's range and each
// point.  Vertex search and projection, row loops -> one loop -> two points
// (us): 300k sites mixed 158 -> 152 -> 151, 50k ref 59 -> 54 -> 52, 100k fp64
// 81 -> 79 -> 73.
template <class T, class PT, int KK, class Accept>
__device__ __forceinline__ bool grid_knn_box(const GridGeom& g, const int* __restrict__ cell_start,
                                             const Pt4<PT>* __restrict__ pts, V3<T> q, T thr, float rad,
                                             TopK<T, KK>& top, Accept accept, int max_cells) {
  if (!finite3(q) || !(rad < INFINITY) || !(thr >= (T)0)) return false;
  const float qf[3] = {(float)q.x, (float)q.y, (float)q.z};
  int lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = grid_coord(g, __fsub_rd(qf[a], rad), a);
    hi[a] = grid_coord(g, __fadd_ru(qf[a], rad), a);
  }
  if ((hi[0] - lo[0] + 1) * (hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1) > max_cells) return false;
  const int ny = hi[1] - lo[1] + 1, rows = (hi[2] - lo[2] + 1) * ny;
  int y = lo[1], row = g.cell_base + (lo[2] * g.dim[1] + lo[1]) * g.dim[0];
  int nk = __ldg(cell_start + row + lo[0]), ne = __ldg(cell_start + row + hi[0] + 1);
  int k = 0, e = 0;
  for (int r = 0;;) {
    while (k >= e && r < rows) {
      k = nk;
      e = ne;
      if (++r < rows) {
        row += g.dim[0];
        if (++y > hi[1]) { y = lo[1]; row += (g.dim[1] - ny) * g.dim[0]; }
        nk = __ldg(cell_start + row + lo[0]);
        ne = __ldg(cell_start + row + hi[0] + 1);
      }
    }
    if (k >= e) break;
    const Pt4<PT> p[2] = {pts[k], pts[min(k + 1, e - 1)]};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const T d = dist2(V3<T>{(T)p[j].x, (T)p[j].y, (T)p[j].z}, q);
      if (k + j < e && accept(p[j].id) && d <= thr && d <= top.worst_d()) top.insert(KeyOps<T>::make(d, p[j].id));
    }
    k += 2;
  }
  return top.full();
}

// ---------------------------------------------------------------------------
// warp-cooperative search: one warp per query point
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long shfl_key(unsigned long long k, int src) {
  return __shfl_sync(0xffffffffu, k, src);
}
__device__ __forceinline__ DKey shfl_key(DKey k, int src) {
  return {__shfl_sync(0xffffffffu, k.d, src), __shfl_sync(0xffffffffu, k.i, src)};
}
__device__ __forceinline__ unsigned long long shfl_up_key(unsigned long long k) {
  return __shfl_up_sync(0xffffffffu, k, 1);
}
__device__ __forceinline__ DKey shfl_up_key(DKey k) {
  return {__shfl_up_sync(0xffffffffu, k.d, 1), __shfl_up_sync(0xffffffffu, k.i, 1)};
}
__device__ __forceinline__ unsigned long long min_key(unsigned long long) { return 0ull; }
__device__ __forceinline__ DKey min_key(DKey) { return {-INFINITY, 0u}; }

// Points of slot `slot` of Chebyshev ring r around (cx,cy,cz): two slots per
// (z,y) row, the whole x-range for rows on the shell's faces, else the two end
// cells.  nslots: slots of the ring.
struct RingSlots {
  int cx, cy, cz, r, x0, x1, y0, z0, ny, nslots;
  __device__ __forceinline__ RingSlots(const GridGeom& g, int cx_, int cy_, int cz_, int r_)
      : cx(cx_), cy(cy_), cz(cz_), r(r_), x0(max(cx_ - r_, 0)), x1(min(cx_ + r_, g.dim[0] - 1)), y0(max(cy_ - r_, 0)),
        z0(max(cz_ - r_, 0)), ny(min(cy_ + r_, g.dim[1] - 1) - y0 + 1),
        nslots(2 * (min(cz_ + r_, g.dim[2] - 1) - z0 + 1) * ny) {}
  __device__ __forceinline__ void range(const GridGeom& g, const int* __restrict__ cell_start, int slot, int& b, int& e) const {
    b = e = 0;
    if (slot >= nslots) return;
    const int rowi = slot >> 1, which = slot & 1;
    const int z = z0 + rowi / ny, y = y0 + rowi % ny;
    const int row = g.cell_base + (z * g.dim[1] + y) * g.dim[0];
    const bool full_row = (r == 1) || abs(z - cz) == r || abs(y - cy) == r;
    if (full_row) {
      if (which == 0) { b = __ldg(cell_start + row + x0); e = __ldg(cell_start + row + x1 + 1); }
    } else {
      const int x = which == 0 ? cx - r : cx + r;
      if (x >= 0 && x < g.dim[0]) { b = __ldg(cell_start + row + x); e = __ldg(cell_start + row + x + 1); }
    }
  }
};

// Visit the points of the lanes' ranges [b, e) in chunks of 32: every lane calls
// visit(pos) the same number of times, pos = a sorted position or -1.  The
// lengths are warp-scanned, and each lane finds the range of its candidate by a
// shuffle binary search over the prefix sums.
template <class Visit>
__device__ __forceinline__ void warp_ranges(int b, int e, int lane, Visit&& visit) {
  const int len = e - b;
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int excl = incl - len;
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  for (int c = 0; c < total; c += 32) {
    const int i = c + lane;
    int lo = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
      const int probe = lo + step;
      const int ex = __shfl_sync(0xffffffffu, excl, probe & 31);
      if (probe < 32 && ex <= i) lo = probe;
    }
    const int rb = __shfl_sync(0xffffffffu, b, lo);
    const int rex = __shfl_sync(0xffffffffu, excl, lo);
    visit(i < total ? rb + (i - rex) : -1);
  }
}

// Visit the candidates of ring r, its slots spread over the lanes.
template <class Visit>
__device__ __forceinline__ void warp_ring(const GridGeom& g, const int* __restrict__ cell_start, int cx, int cy,
                                          int cz, int r, int lane, Visit&& visit) {
  const RingSlots R(g, cx, cy, cz, r);
  for (int base = 0; base < R.nslots; base += 32) {
    int b, e;
    R.range(g, cell_start, base + lane, b, e);
    warp_ranges(b, e, lane, visit);
  }
}

// lower bound on the distance from q to any cell outside ring r (+inf when
// the visited block covers the grid)
__device__ __forceinline__ float ring_margin(const GridGeom& g, const float qf[3], const int c[3], int r) {
  float m = __int_as_float(0x7f800000);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (c[a] - r > 0) m = fminf(m, qf[a] - (g.lo[a] + (float)(c[a] - r) * g.h));
    if (c[a] + r < g.dim[a] - 1) m = fminf(m, (g.lo[a] + (float)(c[a] + r + 1) * g.h) - qf[a]);
  }
  return m;
}

// Exact KK nearest points of q (uniform across the warp), KK <= 64.  The
// sorted list spans R = ceil(KK/32) registers per lane: list[r] at lane j is
// entry 32*r + j.  Candidates beyond the estimate thr0 (the caller's guess of
// the KK-th squared distance) are skipped, and thr tightens to the current
// KK-th distance once the list is full.  The result is exact whatever the
// estimate: a skipped candidate lies above a threshold that is >= the final
// KK-th distance, and an estimate that proves too tight (the list is not full
// although every point within it was visited) restarts the search with
// thr = +inf.
template <class T, class PT, int KK, class Accept>
__device__ __forceinline__ void warp_knn(const GridGeom& g, const int* __restrict__ cell_start,
                                         const Pt4<PT>* __restrict__ pts, V3<T> q, T thr0, int lane, Accept accept,
                                         typename KeyOps<T>::Key (&list)[(KK + 31) / 32]) {
  constexpr int R = (KK + 31) / 32;
  static_assert(KK <= 64, "at most two keys per lane");
  using O = KeyOps<T>;
  using Key = typename O::Key;
#pragma unroll
  for (int r = 0; r < R; ++r) list[r] = O::empty();
  if (!finite3(q)) return;
  const int c[3] = {grid_coord(g, q.x, 0), grid_coord(g, q.y, 1), grid_coord(g, q.z, 2)};
  const float qf[3] = {(float)q.x, (float)q.y, (float)q.z};
  const int rmax = max(g.dim[0], max(g.dim[1], g.dim[2]));
  const float slack = 1e-3f * g.h;
  const T INF = (T)INFINITY;
  constexpr int KR = (KK - 1) / 32, KL = (KK - 1) % 32;  // the K-th entry
  T thr = thr0 > (T)0 ? thr0 : INF;
  Key kth = O::empty();
  for (int ring = 1; ring <= rmax; ++ring) {
    warp_ring(g, cell_start, c[0], c[1], c[2], ring, lane, [&](int pos) {
      Key key = O::empty();
      bool pass = false;
      if (pos >= 0) {
        const Pt4<PT> p = pts[pos];
        if (accept(p.id)) {
          const T d = dist2(V3<T>{(T)p.x, (T)p.y, (T)p.z}, q);
          key = O::make(d, p.id);
          pass = d <= thr && O::less(key, kth);
        }
      }
      unsigned mask = __ballot_sync(0xffffffffu, pass);
      if (mask) {
        while (mask) {
          const int src = __ffs(mask) - 1;
          mask &= mask - 1;
          const Key x = shfl_key(key, src);
          // new[j] = max(old[j-1], min(old[j], x)) over the whole list.  A key
          // that is no longer below the K-th entry leaves entries < KK
          // unchanged, so the K-th entry is refreshed once per chunk; lanes
          // past the list's end hold overflow entries that are never read.
          Key carry = min_key(x);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            Key prev = shfl_up_key(list[r]);
            if (lane == 0) prev = carry;
            if (r + 1 < R) carry = shfl_key(list[r], 31);
            list[r] = O::kmax(prev, O::kmin(list[r], x));
          }
        }
        kth = shfl_key(list[KR], KL);
      }
    });
    const bool full = !O::is_empty(kth);
    if (full) thr = fmin(thr, O::dist(kth));
    float m = ring_margin(g, qf, c, ring);
    const bool all_seen = isinf(m);
    m -= slack;
    if (full) {
      if (all_seen || (m > 0.f && (double)O::dist(kth) < (double)m * (double)m)) break;
    } else if (thr < INF && (all_seen || (m > 0.f && (double)thr < (double)m * (double)m))) {
      thr = INF;
#pragma unroll
      for (int r = 0; r < R; ++r) list[r] = O::empty();
      kth = O::empty();
      ring = 0;
    } else if (all_seen) {
      break;
    }
  }
}

// ---------------------------------------------------------------------------
// Radius query + sort: one warp per query point
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long shfl_xor_key(unsigned long long k, int m) {
  return __shfl_xor_sync(0xffffffffu, k, m);
}
__device__ __forceinline__ DKey shfl_xor_key(DKey k, int m) {
  return {__shfl_xor_sync(0xffffffffu, k.d, m), __shfl_xor_sync(0xffffffffu, k.i, m)};
}

// Bitonic sort of 64 keys held two per lane (element 32 r + lane in k[r]),
// ascending: 21 compare-exchange steps, all but one across lanes.
template <class T>
__device__ __forceinline__ void warp_bitonic64(typename KeyOps<T>::Key (&k)[2], int lane) {
  using O = KeyOps<T>;
#pragma unroll
  for (int kk = 2; kk <= 64; kk <<= 1) {
#pragma unroll
    for (int j = kk >> 1; j > 0; j >>= 1) {
      if (j == 32) {  // kk == 64: the partner is the lane's other register, ascending
        const auto lo = O::kmin(k[0], k[1]), hi = O::kmax(k[0], k[1]);
        k[0] = lo; k[1] = hi;
      } else {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const bool up = ((32 * r + lane) & kk) == 0;
          const auto o = shfl_xor_key(k[r], j);
          k[r] = (((lane & j) == 0) == up) ? O::kmin(k[r], o) : O::kmax(k[r], o);
        }
      }
    }
  }
}

// Sort of the first cnt <= 64 keys of buf into list (element 32 r + lane in
// list[r]), ascending.  The bitonic network runs on 32-bit words, 26 bits of
// the squared distance scaled by thr >= every distance and the key's place in
// buf; two distances that agree in those bits leave two keys out of order (a
// few per cent of the searches), which the check finds and the full-width
// network puts right.
template <class T>
__device__ __forceinline__ void warp_sort64(const typename KeyOps<T>::Key* buf, int cnt, T thr, int lane,
                                            typename KeyOps<T>::Key (&list)[2]) {
  using O = KeyOps<T>;
  const float scale = 67108863.f / (float)thr;
  uint32_t w[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int e = 32 * r + lane;
    w[r] = 0xffffffffu;
    if (e < cnt) w[r] = (min((uint32_t)((float)O::dist(buf[e]) * scale), 0x3fffffeu) << 6) | (uint32_t)e;
  }
#pragma unroll
  for (int kk = 2; kk <= 64; kk <<= 1) {
#pragma unroll
    for (int j = kk >> 1; j > 0; j >>= 1) {
      if (j == 32) {
        const uint32_t lo = min(w[0], w[1]), hi = max(w[0], w[1]);
        w[0] = lo; w[1] = hi;
      } else {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const bool up = ((32 * r + lane) & kk) == 0;
          const uint32_t o = __shfl_xor_sync(0xffffffffu, w[r], j);
          w[r] = (((lane & j) == 0) == up) ? min(w[r], o) : max(w[r], o);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) list[r] = w[r] == 0xffffffffu ? O::empty() : buf[w[r] & 63u];
  const auto p0 = shfl_up_key(list[0]), p1 = shfl_up_key(list[1]), last = shfl_key(list[0], 31);
  const bool off = (lane > 0 && O::less(list[0], p0)) || O::less(list[1], lane > 0 ? p1 : last);
  if (__any_sync(0xffffffffu, off)) warp_bitonic64<T>(list, lane);
}

// Exact MM nearest points of q (uniform across the warp) from one radius
// query: every accepted point whose squared distance is <= thr is gathered
// into buf (the warp's kRadiusKeys keys of shared memory); of more than 64
// only those within a smaller threshold that still holds MM are kept (counted
// by ballots; the count grows in proportion to the squared distance, so the
// first guess usually does), and the rest are sorted.  The first MM of list
// (element 32 r + lane in list[r], the layout of warp_knn) are the MM nearest
// in (squared distance, index) order: every point left out is farther than
// every key kept.  The cells visited are those of the box q +- rad, which the
// caller sizes so that it holds every point within sqrt(thr) (rad rounded up
// with margin; cell coordinates are monotone in the position).  Returns false
// when fewer than MM or more than kRadiusKeys points pass, or no threshold
// separates MM to 64 of them (equal distances); the caller then runs warp_knn.
//
// (With 64 keys and no second threshold 27 % of the searches for 48 of 1M
// random sites fell back to the ring search, at three to five times the cost:
// all 1M sites in 2.93 ms, now 1.97 at 1200 warp instructions per search; the
// 130k to 400k searches of the next iterations 0.30 to 0.80 -> 0.24 to 0.75.)
constexpr int kRadiusKeys = 128;

template <class T, class PT, int MM, class Accept>
__device__ __forceinline__ bool warp_radius_knn(const GridGeom& g, const int* __restrict__ cell_start,
                                                const Pt4<PT>* __restrict__ pts, V3<T> q, T thr, float rad,
                                                int lane, Accept accept, typename KeyOps<T>::Key* buf,
                                                typename KeyOps<T>::Key (&list)[2]) {
  static_assert(MM >= 1 && MM <= 60, "MM to 64 neighbours are sorted");
  using O = KeyOps<T>;
  using Key = typename O::Key;
  if (!finite3(q) || !(rad < INFINITY) || !(thr > (T)0)) return false;
  const float qf[3] = {(float)q.x, (float)q.y, (float)q.z};
  int lo[3], hi[3];
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    lo[ax] = grid_coord(g, __fsub_rd(qf[ax], rad), ax);
    hi[ax] = grid_coord(g, __fadd_ru(qf[ax], rad), ax);
  }
  const int ny = hi[1] - lo[1] + 1;
  const int nrows = ny * (hi[2] - lo[2] + 1);
  // lower bound on the distance along axis a from q to the points of cell
  // layer c (the edge layers also hold the points beyond the grid)
  auto beyond = [&](float v, int c, int a) {
    const float l = g.lo[a] + (float)c * g.h;
    const float below = c > 0 ? l - v : 0.f, above = c < g.dim[a] - 1 ? v - (l + g.h) : 0.f;
    return fmaxf(fmaxf(below, above) - 2e-3f * g.h - 4e-7f * fabsf(v), 0.f);
  };
  const unsigned below = (1u << lane) - 1u;
  int cnt = 0;
  for (int base = 0; base < nrows; base += 32) {
    // one (z, y) row of the box per lane: the contiguous range of sorted points
    // of the cells that the ball of radius rad reaches in it
    const int rowi = base + lane;
    int b = 0, e = 0;
    if (rowi < nrows) {
      const int z = lo[2] + rowi / ny, y = lo[1] + rowi % ny;
      const float fy = beyond(qf[1], y, 1), fz = beyond(qf[2], z, 2);
      const float rx2 = rad * rad * 1.0001f - fy * fy - fz * fz;
      if (rx2 >= 0.f) {
        const float rx = fminf(__fsqrt_ru(rx2) * 1.0001f + 1e-3f * g.h, rad);
        const int row = g.cell_base + (z * g.dim[1] + y) * g.dim[0];
        b = __ldg(cell_start + row + grid_coord(g, __fsub_rd(qf[0], rx), 0));
        e = __ldg(cell_start + row + grid_coord(g, __fadd_ru(qf[0], rx), 0) + 1);
      }
    }
    unsigned filled = __ballot_sync(0xffffffffu, b < e);
    // the rows' points in chunks of 32, each chunk loaded while the one before
    // it is looked at
    int i = 0, re = 0;
    bool more = filled != 0u;
    Pt4<PT> next{};
    auto advance = [&]() {
      if (i - lane + 32 < re) {
        i += 32;
      } else if (filled) {
        const int src = __ffs(filled) - 1;
        filled &= filled - 1;
        i = __shfl_sync(0xffffffffu, b, src) + lane;
        re = __shfl_sync(0xffffffffu, e, src);
      } else {
        more = false;
        return;
      }
      if (i < re) next = pts[i];
    };
    if (more) advance();
    while (more) {
      const Pt4<PT> p = next;
      const bool in = i < re;
      advance();
      bool pass = false;
      Key key = O::empty();
      if (in && accept(p.id)) {
        const T d = dist2(V3<T>{(T)p.x, (T)p.y, (T)p.z}, q);
        key = O::make(d, p.id);
        pass = d <= thr;
      }
      const unsigned m = __ballot_sync(0xffffffffu, pass);
      const int slot = cnt + __popc(m & below);
      if (pass && slot < kRadiusKeys) buf[slot] = key;
      cnt += __popc(m);
      if (cnt > kRadiusKeys) return false;
    }
  }
  if (cnt < MM) return false;
  __syncwarp();
  if (cnt > 64) {
    constexpr int R = kRadiusKeys / 32;
    Key k[R];
    T d[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      k[r] = 32 * r + lane < cnt ? buf[32 * r + lane] : O::empty();
      d[r] = O::dist(k[r]);  // empty: +inf
    }
    T dlo = (T)0, dhi = thr, t = thr * (T)((MM + 64) / 2.0) / (T)cnt;
    int n = 0;
    for (int it = 0; it < 12; ++it) {
      n = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) n += __popc(__ballot_sync(0xffffffffu, d[r] <= t));
      if (n >= MM && n <= 64) break;
      if (n < MM) dlo = t; else dhi = t;
      t = (dlo + dhi) * (T)0.5;
    }
    if (n < MM || n > 64) return false;
    thr = t;
    cnt = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool pass = d[r] <= t;
      const unsigned m = __ballot_sync(0xffffffffu, pass);
      if (pass) buf[cnt + __popc(m & below)] = k[r];
      cnt += __popc(m);
    }
    __syncwarp();
  }
  warp_sort64<T>(buf, cnt, thr, lane, list);
  __syncwarp();  // every lane has read buf before the next query writes it
  return true;
}

// ---------------------------------------------------------------------------
// grid build: count -> exclusive scan -> scatter
// ---------------------------------------------------------------------------
struct SegGrid {           // the minimal per-point view the build needs
  const GridGeom* geom;    // one geometry per segment
  const int* seg_of;       // segment of each point (nullptr: all segment 0)
};

template <class T>
__global__ void k_grid_count(int n, const T* __restrict__ P, SegGrid sg, int* __restrict__ cell_count,
                             int2* __restrict__ cellrank) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  int cell = grid_cell(sg.geom[sg.seg_of ? sg.seg_of[g] : 0], ld3(P, g));
  int rank = atomicAdd(cell_count + cell, 1);
  cellrank[g] = make_int2(cell, rank);
}

template <class T>
__global__ void k_grid_scatter(int n, const T* __restrict__ P, const int2* __restrict__ cellrank,
                               const int* __restrict__ cell_start, Pt4<T>* __restrict__ sorted) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  int2 cr = cellrank[g];
  V3<T> p = ld3(P, g);
  Pt4<T> o;
  o.x = p.x; o.y = p.y; o.z = p.z; o.id = (uint32_t)g;
  sorted[cell_start[cr.x] + cr.y] = o;
}

// Exclusive scan of n ints: block sums, scan of the block sums, then a
// block-local rescan with the block offset.  out[n] = total.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int block_exclusive_scan(int v, int* smem_warp, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem_warp[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int w = (lane < (blockDim.x >> 5)) ? smem_warp[lane] : 0;
    int ws = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += y;
    }
    smem_warp[lane] = ws - w;
    if (lane == 31) smem_warp[32] = ws;
  }
  __syncthreads();
  total = smem_warp[32];
  int r = smem_warp[wid] + x - v;
  __syncthreads();
  return r;
}

// one block scans the block sums tile by tile, carrying the running total
__device__ __forceinline__ void scan_partials_block(int nb, int* __restrict__ part, int* sw) {
  int carry = 0;
  for (int tile = 0; tile < nb; tile += kScanTile) {
    int base = tile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) { v[k] = (base + k < nb) ? part[base + k] : 0; s += v[k]; }
    int total;
    int off = block_exclusive_scan(s, sw, total) + carry;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (base + k < nb) part[base + k] = off;
      off += v[k];
    }
    carry += total;
  }
  if (threadIdx.x == 0) part[nb] = carry;
}

// Block sums of the input.  With a ticket (a zeroed counter), the last block
// to finish also scans the block sums (the partials step), so the scan takes
// two launches; it leaves the ticket at zero again.
__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(int n, const int* __restrict__ in, int* __restrict__ part,
                                                              unsigned* ticket) {
  __shared__ int sw[33];
  __shared__ bool last;
  int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += (base + k < n) ? in[base + k] : 0;
  int total;
  block_exclusive_scan(s, sw, total);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
  if (ticket == nullptr) return;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  scan_partials_block(gridDim.x, part, sw);
  if (threadIdx.x == 0) *ticket = 0u;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_partials(int nb, int* __restrict__ part) {
  __shared__ int sw[33];
  scan_partials_block(nb, part, sw);
}

// clear_in: the input is zeroed once read (the engine's cell counts are then
// ready for the next iteration's counting without a memset)
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(int n, int* __restrict__ in, const int* __restrict__ part,
                                                             int* __restrict__ out, int clear_in) {
  __shared__ int sw[33];
  int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) { v[k] = (base + k < n) ? in[base + k] : 0; s += v[k]; }
  if (clear_in) {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
      if (base + k < n) in[base + k] = 0;
  }
  int total;
  int off = block_exclusive_scan(s, sw, total) + part[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = off;
    off += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = part[gridDim.x];
}

inline int scan_blocks(int n) { return (n + kScanTile - 1) / kScanTile; }

// part must hold scan_blocks(n) + 1 ints
// Exclusive scan of n ints, out[n] = total.  With a ticket (a zeroed
// counter owned by the caller) two launches, else three; returns the number
// of launches.
inline int launch_exclusive_scan(int n, int* in, int* part, int* out, cudaStream_t st, bool clear_in = false,
                                 unsigned* ticket = nullptr) {
  int nb = scan_blocks(n);
  if (nb < 1) nb = 1;
  k_scan_reduce<<<nb, kScanThreads, 0, st>>>(n, in, part, ticket);
  if (ticket == nullptr) k_scan_partials<<<1, kScanThreads, 0, st>>>(nb, part);
  k_scan_apply<<<nb, kScanThreads, 0, st>>>(n, in, part, out, clear_in ? 1 : 0);
  return ticket == nullptr ? 3 : 2;
}

}  // namespace cvt
