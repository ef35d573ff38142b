// Exact K-nearest search of many neighbouring queries: one query per lane,
// the warp's queries share one walk over the cells around them.
//
// Every lane keeps the places of the candidates within its own radius in a
// column of shared memory; the warp visits the cells of the union of its
// lanes' boxes, so the walk has no divergence and each candidate is one
// broadcast load for 32 queries.  A lane then sorts its own candidates (up to
// 64) in registers: 32-bit words of 26 bits of the squared distance and the
// place in the column, through a fixed network of minima and maxima; words
// that agree in the distance bits send the lane through an insertion pass with
// the full keys.  Queries whose radius holds too few or too many points are
// left to the caller (one warp per query).
//
// Bound by issue: of about 310 warp instructions per query (K = 33) half are
// the walk.  1M points, K = 33: 1.05 ms and 0.10 for the queries left over
// (1.25 with the grid build); a sorted list per thread in registers, one
// insertion per accepted candidate of any lane, took 2.17.  (Tried for the engine's full searches too: its cells,
// sized for K + 1 sites, make the union walk twice as long, no faster than a
// warp per site.)
#pragma once
#include <climits>
#include "cvt_grid.cuh"

namespace cvt {

constexpr int kGroupReach = 4;   // cells between a group's leader and its members
constexpr int kGroupCap = 64;

// One warp's columns: places (in the cell-ordered points) of each lane's
// candidates; a column of padding keeps a warp that reads one lane's column (a
// row store) free of conflicts.
struct GroupPlaces { int at[kGroupCap][33]; };

// Batcher's odd-even merge sort of N words in registers.
__device__ __forceinline__ void sort2(uint32_t& a, uint32_t& b) {
  const uint32_t lo = min(a, b), hi = max(a, b);
  a = lo; b = hi;
}
template <int LO, int LEN, int R, int N> __device__ __forceinline__ void merge_words(uint32_t (&w)[N]) {
  if constexpr (2 * R < LEN) {
    merge_words<LO, LEN, 2 * R>(w);
    merge_words<LO + R, LEN, 2 * R>(w);
#pragma unroll
    for (int i = LO + R; i + R < LO + LEN; i += 2 * R) sort2(w[i], w[i + R]);
  } else {
    sort2(w[LO], w[LO + R]);
  }
}
template <int LO, int LEN, int N> __device__ __forceinline__ void sort_words(uint32_t (&w)[N]) {
  if constexpr (LEN > 1) {
    sort_words<LO, LEN / 2>(w);
    sort_words<LO + LEN / 2, LEN / 2>(w);
    merge_words<LO, LEN, 1>(w);
  }
}

// Radius of a box query that covers every point within squared distance thr.
__device__ __forceinline__ float query_radius(const GridGeom& g, V3<float> q, float thr_ru) {
  const float qm = fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z)));
  return __fsqrt_ru(thr_ru) * 1.0001f + 1e-3f * g.h + 4e-7f * qm;
}

// For each lane with valid set: the points within squared distance thr of q;
// afterwards the lane's column holds their places, the first `want` of them the
// nearest in (distance, id) order.  Returns whether the lane's query is
// answered: at least want and at most kGroupCap points within thr.  Every point
// left out is farther than every one held.  Warp-collective.
__device__ __forceinline__ bool group_knn(const GridGeom& g, const int* __restrict__ cell_start,
                                          const Pt4<float>* __restrict__ pts, bool valid, V3<float> q, float thr,
                                          float rad, int want, GroupPlaces& L) {
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  valid = valid && finite3(q) && rad < INFINITY && thr > 0.f;
  int at[3], lo[3], hi[3];
  {
    const float qf[3] = {q.x, q.y, q.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      at[a] = valid ? grid_coord(g, qf[a], a) : 0;
      lo[a] = valid ? grid_coord(g, __fsub_rd(qf[a], rad), a) : 0;
      hi[a] = valid ? grid_coord(g, __fadd_ru(qf[a], rad), a) : 0;
    }
  }
  valid = valid && hi[0] - lo[0] <= 8 && hi[1] - lo[1] <= 8 && hi[2] - lo[2] <= 8;
  int cnt = 0;
  for (unsigned pending = __ballot_sync(full, valid); pending;) {
    const int leader = __ffs(pending) - 1;
    bool member = ((pending >> lane) & 1u) != 0u;
#pragma unroll  // (every lane takes part in every shuffle)
    for (int a = 0; a < 3; ++a) {
      const int la = __shfl_sync(full, at[a], leader);
      member = member && abs(at[a] - la) <= kGroupReach;
    }
    pending &= ~__ballot_sync(full, member);
    int ulo[3], uhi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      ulo[a] = __reduce_min_sync(full, member ? lo[a] : INT_MAX);
      uhi[a] = __reduce_max_sync(full, member ? hi[a] : INT_MIN);
    }
    const int ny = uhi[1] - ulo[1] + 1, nrows = ny * (uhi[2] - ulo[2] + 1);
    for (int r0 = 0; r0 < nrows; r0 += 32) {
      const int r = r0 + lane;
      int b = 0, e = 0;
      if (r < nrows) {
        const int row = g.cell_base + ((ulo[2] + r / ny) * g.dim[1] + ulo[1] + r % ny) * g.dim[0];
        b = __ldg(cell_start + row + ulo[0]);
        e = __ldg(cell_start + row + uhi[0] + 1);
      }
      unsigned filled = __ballot_sync(full, b < e);
      while (filled) {
        const int src = __ffs(filled) - 1;
        filled &= filled - 1;
        const int re = __shfl_sync(full, e, src);
        int i = __shfl_sync(full, b, src);
        auto look = [&](const Pt4<float>& p, int place) {
          // (before the condition: behind `member`, all 1M searches take 11 % longer)
          const float d = dist2(V3<float>{p.x, p.y, p.z}, q);
          if (member && d <= thr) {
            if (cnt < kGroupCap) L.at[cnt][lane] = place;
            ++cnt;
          }
        };
        for (; i + 4 <= re; i += 4) {
          Pt4<float> p[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) p[k] = pts[i + k];
#pragma unroll
          for (int k = 0; k < 4; ++k) look(p[k], i + k);
        }
        for (; i < re; ++i) look(pts[i], i);
      }
    }
  }
  const bool ok = valid && cnt >= want && cnt <= kGroupCap;
  if (__any_sync(full, ok)) {
    const int n = ok ? cnt : 0;
    const float scale = 67108863.f / thr;
    uint32_t w[kGroupCap];
#pragma unroll
    for (int k = 0; k < kGroupCap; ++k) {
      w[k] = 0xffffffffu;
      if (k < n) {
        const Pt4<float> p = pts[L.at[k][lane]];
        const float d = dist2(V3<float>{p.x, p.y, p.z}, q);
        w[k] = (min((uint32_t)(d * scale), 0x3fffffeu) << 6) | (uint32_t)k;
      }
    }
    sort_words<0, kGroupCap>(w);
    bool tie = false;
#pragma unroll
    for (int k = 0; k + 1 < kGroupCap; ++k) tie = tie || (k < want && k + 1 < n && (w[k] >> 6) == (w[k + 1] >> 6));
#pragma unroll
    for (int k = 0; k < kGroupCap; ++k)
      if (k < n) w[k] = (uint32_t)L.at[w[k] & 63u][lane];
#pragma unroll
    for (int k = 0; k < kGroupCap; ++k)
      if (k < n) L.at[k][lane] = (int)w[k];
    if (tie) {
      auto key = [&](int place, float& d, uint32_t& id) {
        const Pt4<float> p = pts[place];
        d = dist2(V3<float>{p.x, p.y, p.z}, q);
        id = p.id;
      };
      for (int t = 1; t < n; ++t) {
        const int place = L.at[t][lane];
        float d;
        uint32_t id;
        key(place, d, id);
        int s = t;
        for (; s > 0; --s) {
          const int before = L.at[s - 1][lane];
          float db;
          uint32_t ib;
          key(before, db, ib);
          if (db < d || (db == d && ib < id)) break;
          L.at[s][lane] = before;
        }
        L.at[s][lane] = place;
      }
    }
  }
  __syncwarp();
  return ok;
}

// The k <= 32 R nearest of q by one warp, ring by ring as in warp_knn
// (cvt_grid.cuh) with a run-time k, from ring `first` on (list: the nearest of
// the rings before it; empty for first = 1).  far > 0: a query whose rings take
// more than far look-ups of cell ranges scans all n_pts points instead; at once
// when its distance from the grid alone asks for so many.
template <class T, class PT, int R, class Accept>
__device__ __forceinline__ void warp_knn_k(const GridGeom& g, const int* __restrict__ cell_start,
                                           const Pt4<PT>* __restrict__ pts, int n_pts, V3<T> q, int k, int lane,
                                           Accept accept, int first, float far, typename KeyOps<T>::Key (&list)[R]) {
  using O = KeyOps<T>;
  using Key = typename O::Key;
  if (!finite3(q)) return;
  auto last_key = [&]() { return shfl_key((k - 1) / 32 == 0 ? list[0] : list[R - 1], (k - 1) % 32); };
  Key kth = last_key();
  auto look = [&](bool in, const Pt4<PT>& p) {
    Key key = O::empty();
    bool pass = false;
    if (in && accept(p.id)) {
      key = O::make(dist2(V3<T>{(T)p.x, (T)p.y, (T)p.z}, q), p.id);
      pass = O::less(key, kth);
    }
    unsigned mask = __ballot_sync(0xffffffffu, pass);
    if (!mask) return;
    while (mask) {
      const int src = __ffs(mask) - 1;
      mask &= mask - 1;
      const Key x = shfl_key(key, src);
      Key carry = min_key(x);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        Key prev = shfl_up_key(list[r]);
        if (lane == 0) prev = carry;
        if (r + 1 < R) carry = shfl_key(list[r], 31);
        list[r] = O::kmax(prev, O::kmin(list[r], x));
      }
    }
    kth = last_key();
  };
  auto visit = [&](int pos) { look(pos >= 0, pts[max(pos, 0)]); };
  const int c[3] = {grid_coord(g, q.x, 0), grid_coord(g, q.y, 1), grid_coord(g, q.z, 2)};
  const float qf[3] = {(float)q.x, (float)q.y, (float)q.z};
  const int rmax = max(g.dim[0], max(g.dim[1], g.dim[2]));
  // ranges that warp_ring looks up in ring r: two per row
  auto ranges = [&](int r) {
    return 2.f * (float)((min(c[1] + r, g.dim[1] - 1) - max(c[1] - r, 0) + 1) *
                         (min(c[2] + r, g.dim[2] - 1) - max(c[2] - r, 0) + 1));
  };
  float looked = 0.f;
  if (far > 0.f) {
    float out2 = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float d = fmaxf(fmaxf(g.lo[a] - qf[a], qf[a] - (g.lo[a] + (float)g.dim[a] * g.h)), 0.f);
      out2 = fmaT(d, d, out2);
    }
    const int rings = (int)fminf(__fsqrt_rn(out2) * g.inv_h, (float)rmax);
    if ((float)rings * ranges(rings) > 3.f * far) looked = INFINITY;
  }
  for (int ring = first; !(looked > far) && ring <= rmax; ++ring) {
    const RingSlots slots(g, c[0], c[1], c[2], ring);
    for (int s0 = 0; s0 < slots.nslots; s0 += 32) {
      int b, e;
      slots.range(g, cell_start, s0 + lane, b, e);
      if (__any_sync(0xffffffffu, b < e)) warp_ranges(b, e, lane, visit);  // (most of a far ring's are empty)
    }
    const float m = ring_margin(g, qf, c, ring) - 1e-3f * g.h;
    if (isinf(m)) return;
    if (!O::is_empty(kth) && m > 0.f && (double)O::dist(kth) < (double)m * (double)m) return;
    if (far > 0.f) looked += ranges(ring);
  }
  if (!(looked > far)) return;
#pragma unroll
  for (int r = 0; r < R; ++r) list[r] = O::empty();
  kth = O::empty();
  // A lone far query waits for its own loads: four points per lane at a time (a
  // Lloyd step's stages with a few far centroids take 0.91 of the time with one).
  constexpr int kAhead = 4;
  for (int b = lane; b - lane < n_pts; b += 32 * kAhead) {
    Pt4<PT> p[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) p[j] = pts[min(b + 32 * j, n_pts - 1)];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) look(b + 32 * j < n_pts, p[j]);
  }
}

}  // namespace cvt
