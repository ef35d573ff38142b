// Fused Lloyd-iteration kernels over many (mesh, site set) segments.
//
// One iteration (main.cu:669-881 per segment) is:
//   k_site_count the cells of the sites of active segments, and the list of
//                the non-frozen ones
//   grid build   scan -> scatter, on a second stream beside k_knn_verify
//   k_frame_vertex the mesh vertex nearest to each of them (its normal
//                gives the frame, main.cu:685-700), on the second stream
//                while the site KNN runs
//   k_knn_verify per active site (one thread): the K-list from the site's
//                candidate list where its motion bound proves it exact
//   k_knn_search the other active sites (one warp each): exact (K+1)-NN in
//                the segment, drop self (site_knn.cuh:79), by one radius
//                query where a bound is known, else ring by ring; frozen
//                sites keep the previous list (main.cu:678)
//   k_site_clip  per site (one thread): frame (site_normals.cuh:69; or,
//                as an option, from the PCA normal of the neighbours),
//                tangent-plane clip and centroid (2dClip.cuh:82)
//   k_clip_overflow  the same for the rare cells whose polygon outgrows
//                the shared-memory buffer (exact 64-vertex cap)
//   k_site_vsearch per site (one thread): centroid -> 5 nearest vertices
//                (main.cu:719-735, frozen sites keep theirs)
//   k_site_proj  per site (one thread): one-ring projection over those
//                vertices (near_project.cuh:149; or, as an
//                option, the exact closest point through the BVH), freeze test
//                and apply (freezetest.cuh:155-212, 270-327, 451-466),
//                tier assignment on the segment's first iteration
//                (main.cu:640-667)
//   k_site_far   the sites whose centroid lies so far off the surface that
//                the vertex grid search gave up: exact brute-force 5-NN by
//                a block, then the rest of the step
//   (bookkeeping) per-segment iteration counters / statistics slots, run by
//                the last block of k_site_far
// All sizes come from device memory, so the whole iteration is captured once
// in a CUDA graph and relaunched while segments come and go.
//
// Site order.  A segment's sites are stored in the cell order of its grid at
// the time it was placed ("internal" order; a Lloyd run moves sites by less
// than a few cells, so neighbours in space stay neighbours in memory), with
// the caller's index kept beside the position (Pt4::id) and the way back in
// internal_of.  Every per-site kernel then reads and writes consecutive
// sites, and a neighbour gather is one aligned 16-byte load (32 bytes in
// FP64) from lines that its block has just read.  Ties are always broken by
// the caller's indices, so no result depends on the internal order.  The
// per-site lists are stored entry by entry (entry e of site g at
// [e * stride + g]): one thread per site reads them coalesced.  With 12-byte
// positions and row-major lists in the caller's order the gathers went to L2:
// the 25-iteration run of 1M sites (K = 32, mixed) took 53.6 ms, with this
// layout and the list check below 40.2; 100k sites, 100 iterations 23.7 and
// 16.1 ms.
#pragma once
#include "cvt_grid.cuh"

namespace cvt {

constexpr int kStatsRing = 256;   // iterations of per-segment statistics kept
constexpr int kStatsWords = 8;    // same, low, both, newly, maxdisp2 bits, iter, KNN lists reused, searched
constexpr int kKProj = 5;         // KPROJ (main.cu:394)
// Largest box (in vertex-grid cells) a bounded vertex query visits before it
// leaves the site to the ring search: ring 1's 27 cells.
constexpr int kVertexBoxCells = 27;
constexpr int kFallbackCap = 66;  // 64-vertex reference cap + room for the overshoot
// threads per SM that k_site_clip's launch bounds ask to keep resident,
// whatever the block size (polygon buffers: 16 KB per block): 64 registers
// for FP32 polygons (1024 threads; mixed, 300k sites: 57.7 us, 65.5 with 768
// and 80 registers, 66.3 with 896)
constexpr int kClipThreadsF = 1024;
constexpr int kClipThreadsD = 384;

struct MeshDev {
  const float* V;
  const int* F;
  const int* vf_off;
  const int* vf_faces;
  const float* N;
  const int* vcell_start;
  const Pt4<float>* vsorted;
  const float4* ring_head;  // one-ring records, one head and kRingBody body words per CSR entry
  const float4* ring_body;  // (k_build_ring_records)
  BvhView bvh;  // over the faces (built before a segment that projects through it is placed)
  GridGeom vg;
  int nV, nF;
  float R;     // clip square half-size: longest input bbox edge (main.cu:421)
  float thr2;  // freeze displacement threshold, squared (main.cu:431)
};

struct SegDev {
  int mesh;       // index into the mesh table
  int site_base;  // first global site index
  int n_sites;
  int mode;       // 0 / 1 / 2
  int ex_quirk;
  int iter;       // iterations completed (device-side count)
  float kth_est;  // first-iteration estimate of the K-th neighbour's squared distance
  float stop_motion2;  // stop once an iteration's max squared motion <= this (< 0: never)
  int stop_iters;      // stop after this many iterations (0: never)
  float thr2_tier[6];
  int need_tier[6];
  float step_motion;   // largest site motion of the segment's last iteration
  int p0;              // buffer parity when the segment was placed
};

template <int PROF> struct PT;
template <> struct PT<PROF_REF> { using T = float; using Q = float; using PP = float; };
template <> struct PT<PROF_MIXED> { using T = float; using Q = double; using PP = float; };
template <> struct PT<PROF_FP64> { using T = double; using Q = double; using PP = double; };

template <class T> struct EngineArgs {
  const SegDev* segs;
  const GridGeom* geom;
  const int* active;      // 0 free, 1 iterating, 2 stopped by its stop rule
  const MeshDev* meshes;
  const int* site_seg;
  Pt4<T>* S[2];               // positions in internal order, id = the site's caller index (+ site_base)
  const uint32_t* internal_of;  // the way back: internal index of caller index (+ site_base)
  size_t stride;              // sites the engine holds: entry e of site g's list at [e * stride + g]
  // Neighbour list per site (internal indices, 0xffffffff: none): the K
  // nearest in order, and with candidate lists (MM > 0) MM - K further ones
  // in no order; the K-list is the candidate list's head.
  // Entry e of site g at [g * list_site + e * list_entry]: entry by entry with
  // candidate lists, where most lists are read and rewritten by one thread per
  // site (k_knn_verify); a row per site without, where a warp writes each list
  // in every iteration (100k sites, K = 24: full searches 196 us entry by entry,
  // 152 as rows, the clip 26 and 24).
  uint32_t* list;
  size_t list_site, list_entry;
  uint8_t* same;      // list unchanged vs the previous iteration (site KNN kernels)
  float* kth;         // last K-th neighbour's squared distance per site, < 0 unknown
  int* act;           // the sites whose list is recomputed
  int* act_count;
  int* knnv;          // 5 nearest vertices, entry k of site g at [k * stride + g]
  int* nnv;
  uint8_t* frozen;
  uint8_t* streak;
  uint8_t* tier;
  const int* cell_start;
  const Pt4<T>* sorted;  // cell-ordered copy of the positions, id = caller index (+ site_base)
  int* stats;
  int* ovf;  // [0] = count, [1 + k] = overflowed site
  int* far;  // [0] = count, [1 + k] = site whose vertex search was deferred
  T* cent;   // centroid per site (3 values), k_site_clip -> k_site_proj
  int K;
  int n_sites;    // site slots the launches cover (every placed segment lies below)
  int proj_mode;  // 0: one-ring of the KPROJ nearest vertices; 1: closest point through the BVH
  int* bvh_ovf;   // BVH traversal stack overflows (never expected: the tree depth is bounded)
  float* cand_rho;   // candidate list's MM-th distance when it was built, rounded down (< 0: no list; inf: every other site)
  float* cand_D;     // motion bound accumulated since it was built (k_knn_verify)
  int* srch;         // [0] = count, [1 + k] = site left for a full search
  float* srch_thr;   // [k]: squared distance that the site's MM nearest lie within (< 0: unknown)
  unsigned long long* blockmax;  // per coarse block (cell slots of the segment): iteration << 32 | max motion bits
};

// Segment of site g when its segment is iterating, else -1.
template <class T>
__device__ __forceinline__ int active_seg(const EngineArgs<T>& a, int g) {
  if (g >= a.n_sites) return -1;
  const int s = __ldg(a.site_seg + g);
  return s >= 0 && a.active[s] == 1 ? s : -1;
}

__device__ __forceinline__ float f32_ru(float x) { return x; }
__device__ __forceinline__ float f32_ru(double x) { return __double2float_ru(x); }
__device__ __forceinline__ float f32_rd(float x) { return x; }
__device__ __forceinline__ float f32_rd(double x) { return __double2float_rd(x); }

// Coarse motion blocks of a segment: kBlockCells^3 grid cells, stored in the
// first cells of the segment's cell range (there are fewer blocks than
// cells).  Positions outside the grid fall in the edge blocks, like cells.
// Larger blocks make the step condition looser but take the maximum motion
// over more sites (measured: 4 cells kept more lists than 3 cells of a grid
// sized for the candidate list's length).
constexpr int kBlockCells = 4;
__device__ __forceinline__ int block_dim(const GridGeom& g, int a) { return (g.dim[a] + kBlockCells - 1) / kBlockCells; }

template <class T>
__device__ __forceinline__ int motion_block(const GridGeom& g, V3<T> p, int& bx, int& by, int& bz) {
  bx = grid_coord(g, p.x, 0) / kBlockCells; by = grid_coord(g, p.y, 1) / kBlockCells;
  bz = grid_coord(g, p.z, 2) / kBlockCells;
  return g.cell_base + (bz * block_dim(g, 1) + by) * block_dim(g, 0) + bx;
}

// polygon storage: vertex k at p[k * stride] (shared memory: thread-
// interleaved; local memory: stride 1)
template <class PP> struct PolyRef {
  V2<PP>* p;
  int stride;
  __device__ __forceinline__ V2<PP> get(int k) const { return p[k * stride]; }
  __device__ __forceinline__ void set(int k, V2<PP> v) const { p[k * stride] = v; }
};

// Sutherland-Hodgman clip by a*x + b*y - c <= eps (2dClip.cuh:11-53).  Stops
// with ovf = true before writing vertex `cap` (buffer full); keeps the
// reference's 64-vertex cap (2dClip.cuh:47-50) for larger buffers.  r2 returns
// the largest squared vertex radius of the output (NaN if any vertex is NaN).
template <class PP, class Q>
__device__ __forceinline__ int clip_poly(const PolyRef<PP>& in, int n, const PolyRef<PP>& out, Q a, Q b, Q c,
                                         Q eps, int cap, bool& ovf, Q& r2) {
  r2 = (Q)0;
  if (n <= 0) return 0;
  auto f = [&](V2<PP> p) -> Q { return fmaT(a, (Q)p.x, fmaT(b, (Q)p.y, -c)); };
  auto isect = [&](V2<PP> s, V2<PP> e, Q fs, Q fe) -> V2<PP> {
    Q t = divT(fs, (fs - fe) + (Q)1e-30);
    return {(PP)fmaT(t, (Q)e.x - (Q)s.x, (Q)s.x), (PP)fmaT(t, (Q)e.y - (Q)s.y, (Q)s.y)};
  };
  auto put = [&](int k, V2<PP> v) {
    out.set(k, v);
    const Q q = fmaT((Q)v.y, (Q)v.y, (Q)v.x * (Q)v.x);
    r2 = (q > r2 || q != q) ? q : r2;
  };
  V2<PP> s = in.get(n - 1);
  Q fs = f(s);
  bool ins_s = fs <= eps;
  int m = 0;
  for (int i = 0; i < n; ++i) {
    V2<PP> e = in.get(i);
    Q fe = f(e);
    bool ins_e = fe <= eps;
    if (ins_e) {
      if (!ins_s) {
        if (m >= cap) { ovf = true; return m; }
        put(m++, isect(s, e, fs, fe));
      }
      if (m >= cap) { ovf = true; return m; }
      put(m++, e);
    } else if (ins_s) {
      if (m >= cap) { ovf = true; return m; }
      put(m++, isect(s, e, fs, fe));
    }
    s = e; fs = fe; ins_s = ins_e;
    if (m >= 64) { m = 64; break; }
  }
  return m;
}

// True when the half-plane a*x + b*y <= c holds, as the clip's predicate
// computes it, at every point within sqrt(r2) of the origin: then clipping
// by it returns the polygon unchanged (same vertices, same order) and can be
// skipped.  By Cauchy-Schwarz a*x + b*y <= sqrt((a^2+b^2) r2); the 1e-4
// relative margin covers the rounding of this test (a few ulp) and of the
// predicate fma(a, x, fma(b, y, -c)) (< 2 ulp of c), so the skip is exact.
// c > 1e-18 keeps the products away from underflow.  NaN fails the test.
template <class Q>
__device__ __forceinline__ bool halfplane_contains_disk(Q a, Q b, Q c, Q r2) {
  return c > (Q)1e-18 && fmaT(a, a, b * b) * r2 * (Q)1.0001 < c * c;
}

// Upper bound on ((d.u)^2 + (d.v)^2) / |d|^2 over all d, the largest eigenvalue
// of the frame's Gram matrix by its row sums; at least 1, NaN for a frame with
// NaN (then clip_cell skips nothing).  The stage calls take frames of any length
// and skew from their caller.
__device__ __forceinline__ float frame_gain(V3<float> u, V3<float> v) {
  const float uv = fabsf(dot3(u, v));
  const float x = (dot3(u, u) + uv) * 1.00001f, y = (dot3(v, v) + uv) * 1.00001f;
  const float g = x > y ? x : y;
  return x == x && g <= 1.00002f ? 1.f : x == x ? g : x;
}

// Neighbours of a site for clip_cell and pca_normal: id(t) is entry t of its
// list, valid(id) whether it names a site, pos(id) that site's position.
template <class T> struct RowNeighbours {  // row-major list of local indices into an AoS array
  const T* S;
  const uint32_t* row;
  uint32_t n;
  __device__ __forceinline__ uint32_t id(int t) const { return __ldg(row + t); }
  __device__ __forceinline__ bool valid(uint32_t j) const { return j < n; }
  __device__ __forceinline__ V3<T> pos(uint32_t j) const { return ld3(S, (long)j); }
};
template <class T> struct ListNeighbours {  // the engine's lists
  const Pt4<T>* S;
  const uint32_t* own;  // the site's first entry
  size_t step;
  __device__ __forceinline__ uint32_t id(int t) const { return __ldg(own + t * step); }
  __device__ __forceinline__ bool valid(uint32_t j) const { return j != 0xffffffffu; }
  __device__ __forceinline__ V3<T> pos(uint32_t j) const { return ldp(S, j); }
};

// clip_cell in full generality: every clip copies the polygon from one buffer
// to the other.  Run for the cells that clip_cell gives back.
//
// Security radius: a bisector whose half-plane contains the disk around the
// site that holds the current polygon cannot cut it and is skipped
// (halfplane_contains_disk).  When the row is this iteration's K-nearest list
// of the same positions (ascending distance), every later neighbour j has
// |d_j| >= |d_t|; the tangent-plane normal of its bisector is at most |d_j|
// long and its offset is |d_j|^2/2, so once |d_t|^2 > 4 r2 (with a 1e-3
// margin for the distance keys' rounding) none of the remaining bisectors can
// cut the polygon and the loop ends.  Both shortcuts only leave out clips
// that would return their input unchanged: the result is the same bit for
// bit as clipping by all K bisectors.
template <int PROF, class NB>
__device__ __forceinline__ int clip_cell_full(const NB& nb, V3<typename PT<PROF>::T> si, int K,
                                         const Frame<typename PT<PROF>::T>& fr, float R,
                                         PolyRef<typename PT<PROF>::PP>& cur, PolyRef<typename PT<PROF>::PP>& nxt,
                                         int cap, bool row_sorted) {
  using T = typename PT<PROF>::T;
  using Q = typename PT<PROF>::Q;
  using PP = typename PT<PROF>::PP;
  const PP r = (PP)R;
  cur.set(0, {-r, -r}); cur.set(1, {r, -r}); cur.set(2, {r, r}); cur.set(3, {-r, r});
  int n = 4;
  Q r2 = (Q)2 * (Q)r * (Q)r * (Q)1.0001;
  bool ovf = false;
  // the next neighbour's position is loaded while the current one clips
  uint32_t jn = nb.id(0);
  V3<T> sn = nb.valid(jn) ? nb.pos(jn) : si;
  // Every lane runs all K trips; a finished lane only skips their bodies.  A
  // data-dependent `break` lets lanes leave at different trips, and the warp
  // then runs the rest of the site's work in fragments (measured 2x slower).
  bool done = false;
  for (int t = 0; t < K; ++t) {
    if (done) continue;
    const uint32_t j = jn;
    const V3<T> sj = sn;
    if (t + 1 < K) {
      jn = nb.id(t + 1);
      if (nb.valid(jn)) sn = nb.pos(jn);
    }
    if (!nb.valid(j)) continue;
    Q a, b, c;
    if (PROF == PROF_MIXED) {
      V3<double> d{(double)sj.x - (double)si.x, (double)sj.y - (double)si.y, (double)sj.z - (double)si.z};
      V3<double> u = cvt3<double>(fr.u), v = cvt3<double>(fr.v);
      a = (Q)dot3(d, u); b = (Q)dot3(d, v); c = (Q)(0.5 * dot3(d, d));
    } else {
      V3<T> d = sub3(sj, si);
      a = (Q)dot3(d, fr.u); b = (Q)dot3(d, fr.v); c = (Q)((T)0.5 * dot3(d, d));
    }
    if (halfplane_contains_disk(a, b, c, r2)) {
      done = row_sorted && c > (Q)1e-18 && (Q)2.002 * r2 < c;
      continue;
    }
    n = clip_poly<PP, Q>(cur, n, nxt, a, b, c, (Q)1e-12, cap, ovf, r2);
    if (ovf) { n = -1; done = true; continue; }
    PolyRef<PP> tmp = cur; cur = nxt; nxt = tmp;
    if (n == 0) done = true;
  }
  return n;
}

// Clip the square [-R,R]^2 by the bisectors of the listed neighbours in one
// buffer; returns the vertex count (polygon in P) or -1 when the cell has to
// be redone by clip_cell_full: more than `cap` vertices, a clip whose outside
// vertices are not one cyclic run, or a vertex that is not finite.  The
// polygon is the one clip_cell_full computes, bit for bit.
//
// A clip first finds the outside vertices as a bit mask.  None: the polygon is
// unchanged and nothing is written.  One run p..q (the only case for a convex
// polygon): Sutherland-Hodgman keeps the others and puts one intersection
// before and one after them, so two vertices are computed and the rest moves
// by 2 - (run length) slots; the three orders below are those in which its
// loop from vertex 0 emits them.  In the MIXED profile the mask is found in
// FP32 where that decides the FP64 predicate: the FP32 value errs by less than
// 9 u |d| r + 8 u c (u = 2^-24: difference, frame dots, half square and two
// fma), and 2e-6 (|d| r + c) is left to the FP64 predicate itself; FP64
// coefficients are only computed for those vertices and for real cuts.
// `gain` bounds (a^2 + b^2) / |d|^2 (frame_gain; 1 for the engine's frames, whose
// vectors are orthonormal to 1e-6).  Neighbours with |d|^2 > 4 gain r^2 (margin
// 2.5e-3) cannot cut: skipped, and on this iteration's sorted list they end the
// loop (see clip_cell_full).  The FP32 error above grows with sqrt(gain) too.
//
// Bound by issue (63 %) and latency; 24 of 32 threads active.  Clip kernel,
// mixed, 300k sites, K = 24: 57 us and 117 warp instructions per site, against
// 102 us and 187 with two buffers and every vertex clipped in FP64 (15 of 32
// active, conversions 42 % of their pipe).
template <int PROF, class NB>
__device__ __forceinline__ int clip_cell(const NB& nb, V3<typename PT<PROF>::T> si, int K,
                                         const Frame<typename PT<PROF>::T>& fr, float gain, float R,
                                         const PolyRef<typename PT<PROF>::PP>& P, int cap, bool row_sorted) {
  using T = typename PT<PROF>::T;
  using Q = typename PT<PROF>::Q;
  using PP = typename PT<PROF>::PP;
  constexpr bool kFilter = PROF == PROF_MIXED;
  const PP r = (PP)R;
  P.set(0, {-r, -r}); P.set(1, {r, -r}); P.set(2, {r, r}); P.set(3, {-r, r});
  int n = 4;
  float r2 = 2.f * R * R * 1.0001f;
  // the next neighbour's position is loaded while the current one clips
  uint32_t jn = nb.id(0);
  V3<T> sn = nb.valid(jn) ? nb.pos(jn) : si;
  // every lane runs all K trips; see clip_cell_full
  bool done = false;
  for (int t = 0; t < K; ++t) {
    if (done) continue;
    const uint32_t j = jn;
    const V3<T> sj = sn;
    if (t + 1 < K) {
      jn = nb.id(t + 1);
      if (nb.valid(jn)) sn = nb.pos(jn);
    }
    if (!nb.valid(j)) continue;
    const V3<T> d = sub3(sj, si);
    const V3<float> df = cvt3<float>(d);
    const float dd = dot3(df, df);
    if (dd > 4.01f * gain * r2 && dd > 2e-18f && dd < 1e30f) {
      done = row_sorted;
      continue;
    }
    // the half-plane a x + b y - c <= eps as the predicate computes it
    const Q eps = (Q)1e-12;
    Q a, b, c;
    auto exact_plane = [&]() {
      if (kFilter) {
        V3<double> e{(double)sj.x - (double)si.x, (double)sj.y - (double)si.y, (double)sj.z - (double)si.z};
        a = (Q)dot3(e, cvt3<double>(fr.u)); b = (Q)dot3(e, cvt3<double>(fr.v)); c = (Q)(0.5 * dot3(e, e));
      } else {
        a = (Q)dot3(d, fr.u); b = (Q)dot3(d, fr.v); c = (Q)((T)0.5 * dot3(d, d));
      }
    };
    auto f = [&](V2<PP> v) -> Q { return fmaT(a, (Q)v.x, fmaT(b, (Q)v.y, -c)); };
    unsigned out = 0u;
    float rin = 0.f;
    if (kFilter) {
      const float af = (float)dot3(d, fr.u), bf = (float)dot3(d, fr.v), cf = 0.5f * dd;
      float root;
      asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"(dd * r2 * gain));
      const float tol = 2e-6f * (root + cf) + 2e-12f;
      unsigned unsure = 0u;
      for (int i = 0; i < n; ++i) {
        const V2<PP> v = P.get(i);
        const float x = (float)v.x, y = (float)v.y;
        const float g = fmaT(af, x, fmaT(bf, y, -cf));
        if (!(g < -tol)) { if (g > tol) out |= 1u << i; else unsure |= 1u << i; }
        else rin = fmaxf(rin, fmaT(y, y, x * x));
      }
      if (unsure) {
        exact_plane();
        while (unsure) {
          const int i = __ffs(unsure) - 1;
          unsure &= unsure - 1;
          const V2<PP> v = P.get(i);
          const float x = (float)v.x, y = (float)v.y;
          if (f(v) <= eps) rin = fmaxf(rin, fmaT(y, y, x * x)); else out |= 1u << i;
        }
      }
    } else {
      exact_plane();
      for (int i = 0; i < n; ++i) {
        const V2<PP> v = P.get(i);
        if (f(v) <= eps) rin = fmaxf(rin, f32_ru(fmaT(v.y, v.y, v.x * v.x))); else out |= 1u << i;
      }
    }
    if (out == 0u) continue;
    const unsigned all = 0xffffffffu >> (32 - n);
    if (out == all) { n = 0; done = true; continue; }
    const unsigned starts = out & ~((out << 1) | (out >> (n - 1)));  // outside, the vertex before it inside
    const int len = __popc(out), p = __ffs(starts) - 1;
    if ((starts & (starts - 1)) || n - len + 2 > cap) { n = -1; done = true; continue; }
    const int q = p + len - 1 >= n ? p + len - 1 - n : p + len - 1;
    const int ip = p == 0 ? n - 1 : p - 1, iq = q + 1 == n ? 0 : q + 1;
    if (kFilter) exact_plane();
    auto isect = [&](V2<PP> s, V2<PP> e) -> V2<PP> {
      const Q fs = f(s), fe = f(e);
      const Q u = divT(fs, (fs - fe) + (Q)1e-30);
      return {(PP)fmaT(u, (Q)e.x - (Q)s.x, (Q)s.x), (PP)fmaT(u, (Q)e.y - (Q)s.y, (Q)s.y)};
    };
    const V2<PP> enter = isect(P.get(ip), P.get(p));  // before the run
    const V2<PP> leave = isect(P.get(q), P.get(iq));  // after it
    // kept vertices [lo, hi) move by `shift`
    int lo, hi, shift, at_enter, at_leave;
    if (p <= q && q + 1 < n) {  // v0 .. v(p-1), enter, leave, v(q+1) .. v(n-1)
      lo = q + 1; hi = n; shift = 2 - len; at_enter = p; at_leave = p + 1;
    } else {                    // leave, v(q+1) .. v(p-1), enter
      lo = iq; hi = p; shift = 1 - iq; at_enter = n - len + 1; at_leave = 0;
    }
    if (shift > 0) {
      for (int i = hi - 1; i >= lo; --i) P.set(i + shift, P.get(i));
    } else if (shift < 0) {
      for (int i = lo; i < hi; ++i) P.set(i + shift, P.get(i));
    }
    P.set(at_enter, enter);
    P.set(at_leave, leave);
    n += 2 - len;
    auto rad2 = [&](V2<PP> v) { return f32_ru(fmaT(v.y, v.y, v.x * v.x)); };
    const float re = rad2(enter), rl = rad2(leave);
    r2 = fmaxf(rin, fmaxf(re, rl)) * 1.000001f;
    if (!(re < INFINITY) || !(rl < INFINITY)) { n = -1; done = true; }
  }
  return n;
}

// ---------------------------------------------------------------------------
// tiers (main.cu:18-150) in FP64, identical operation order to the host code
// ---------------------------------------------------------------------------
__device__ inline void sym3_eigenvalues_d(const double C[9], double lam[3]) {
  double v[3] = {1.0, 0.0, 0.0};
  for (int it = 0; it < 20; ++it) {
    double w[3] = {C[0] * v[0] + C[1] * v[1] + C[2] * v[2], C[3] * v[0] + C[4] * v[1] + C[5] * v[2],
                   C[6] * v[0] + C[7] * v[1] + C[8] * v[2]};
    double n = __dsqrt_rn(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    if (n < 1e-30) break;
    v[0] = __ddiv_rn(w[0], n); v[1] = __ddiv_rn(w[1], n); v[2] = __ddiv_rn(w[2], n);
  }
  lam[0] = v[0] * (C[0] * v[0] + C[1] * v[1] + C[2] * v[2]) + v[1] * (C[3] * v[0] + C[4] * v[1] + C[5] * v[2]) +
           v[2] * (C[6] * v[0] + C[7] * v[1] + C[8] * v[2]);
  double C2[9];
  for (int i = 0; i < 9; ++i) C2[i] = C[i];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) C2[3 * r + c] -= lam[0] * v[r] * v[c];
  double v2[3] = {0.0, 1.0, 0.0};
  for (int it = 0; it < 20; ++it) {
    double w[3] = {C2[0] * v2[0] + C2[1] * v2[1] + C2[2] * v2[2], C2[3] * v2[0] + C2[4] * v2[1] + C2[5] * v2[2],
                   C2[6] * v2[0] + C2[7] * v2[1] + C2[8] * v2[2]};
    double n = __dsqrt_rn(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    if (n < 1e-30) break;
    v2[0] = __ddiv_rn(w[0], n); v2[1] = __ddiv_rn(w[1], n); v2[2] = __ddiv_rn(w[2], n);
  }
  lam[1] = v2[0] * (C2[0] * v2[0] + C2[1] * v2[1] + C2[2] * v2[2]) + v2[1] * (C2[3] * v2[0] + C2[4] * v2[1] + C2[5] * v2[2]) +
           v2[2] * (C2[6] * v2[0] + C2[7] * v2[1] + C2[8] * v2[2]);
  lam[2] = C[0] + C[4] + C[8] - lam[0] - lam[1];
}

// normal(i) gives the unit normal of site i as float[3]; row(t) the t-th
// listed neighbour of site i, or -1
template <class RowOf, class NormalOf>
__device__ inline int tier_of(int mode, int i, int K, RowOf row, NormalOf normal) {
  const double TH[4] = {0.15, 0.35, 0.55, 0.80};
  float ni[3];
  normal(i, ni);
  double sum = 0.0;
  int cnt = 0;
  for (int j = 0; j < K; ++j) {
    int jj = row(j);
    if (jj < 0) continue;
    float nj[3];
    normal(jj, nj);
    double c = (double)ni[0] * (double)nj[0] + (double)ni[1] * (double)nj[1] + (double)ni[2] * (double)nj[2];
    if (c > 1.0) c = 1.0;
    if (c < -1.0) c = -1.0;
    sum += c;
    cnt++;
  }
  double nv = cnt > 0 ? (1.0 - __ddiv_rn(sum, (double)cnt)) : 0.0;
  double L = 0.0;
  if (mode == 2) {
    double mean[3] = {0, 0, 0};
    int c2 = 0;
    for (int j = 0; j < K; ++j) {
      int jj = row(j);
      if (jj < 0) continue;
      float nj[3];
      normal(jj, nj);
      for (int a = 0; a < 3; ++a) mean[a] += (double)nj[a];
      c2++;
    }
    if (c2 >= 2) {
      for (int a = 0; a < 3; ++a) mean[a] = __ddiv_rn(mean[a], (double)c2);
      double C[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      for (int j = 0; j < K; ++j) {
        int jj = row(j);
        if (jj < 0) continue;
        float nj[3];
        normal(jj, nj);
        double d[3] = {(double)nj[0] - mean[0], (double)nj[1] - mean[1], (double)nj[2] - mean[2]};
        for (int r = 0; r < 3; ++r)
          for (int c = 0; c < 3; ++c) C[3 * r + c] += d[r] * d[c];
      }
      double lam[3];
      sym3_eigenvalues_d(C, lam);
      double tmp;
      if (lam[0] > lam[1]) { tmp = lam[0]; lam[0] = lam[1]; lam[1] = tmp; }
      if (lam[1] > lam[2]) { tmp = lam[1]; lam[1] = lam[2]; lam[2] = tmp; }
      if (lam[0] > lam[1]) { tmp = lam[0]; lam[0] = lam[1]; lam[1] = tmp; }
      if (lam[2] > 1e-30) L = __ddiv_rn(lam[2] - lam[1], lam[2]);
    }
  }
  int t = 0;
  while (t < 4 && nv >= TH[t]) t++;
  if (mode == 2 && t == 4 && L > 0.80) t = 5;
  return t;
}

// ---------------------------------------------------------------------------
// k_site_count: the grid cell of every site of an iterating segment and its
// rank within the cell (the counting half of the counting sort), and the list
// of the sites whose neighbour list is recomputed this iteration (frozen
// sites keep theirs, main.cu:678), in internal order.  Consecutive sites
// mostly share their cell, so a warp adds to a cell once for all its sites
// in it; the list is appended once per block (per-warp atomics on one counter
// serialise).
// ---------------------------------------------------------------------------
constexpr int kCountThreads = 256;

template <class T>
__global__ void __launch_bounds__(kCountThreads) k_site_count(EngineArgs<T> a, int parity, int* __restrict__ cell_count,
                                                              int2* __restrict__ cellrank) {
  __shared__ int warp_base[kCountThreads / 32];
  __shared__ int block_base;
  const int g = blockIdx.x * kCountThreads + threadIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int s = active_seg(a, g);
  int cell = -1;
  bool act = false;
  if (s >= 0) {
    cell = grid_cell(a.geom[s], ldp(a.S[parity], g));
    act = !(a.segs[s].mode != 0 && a.frozen[g]);
  }
  const unsigned peers = __match_any_sync(0xffffffffu, cell);
  const int leader = __ffs(peers) - 1;
  int base = 0;
  if (cell >= 0 && lane == leader) base = atomicAdd(cell_count + cell, __popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (g < a.n_sites) cellrank[g] = make_int2(cell, base + __popc(peers & ((1u << lane) - 1u)));
  const unsigned m = __ballot_sync(0xffffffffu, act);
  if (lane == 0) warp_base[wid] = __popc(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < kCountThreads / 32; ++w) {
      const int c = warp_base[w];
      warp_base[w] = sum;
      sum += c;
    }
    block_base = sum ? atomicAdd(a.act_count, sum) : 0;
  }
  __syncthreads();
  if (act) a.act[block_base + warp_base[wid] + __popc(m & ((1u << lane) - 1u))] = g;
}

// the scattering half: the cell-ordered copy of the positions
template <class T>
__global__ void k_site_scatter(EngineArgs<T> a, int parity, const int2* __restrict__ cellrank, Pt4<T>* __restrict__ sorted) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= a.n_sites) return;
  const int2 cr = cellrank[g];
  if (cr.x < 0) return;
  sorted[__ldg(a.cell_start + cr.x) + cr.y] = a.S[parity][g];
}

// ---------------------------------------------------------------------------
// k_frame_vertex: each listed site's nearest mesh vertex (the frame vertex,
// main.cu:685-700), one thread per site, in the same key order as any other
// search, so the same vertex.  The site's vertex of the last iteration is
// at the squared distance thr from its new position, so the nearest vertex
// lies in the box of cells within sqrt(thr): a few cells, against the 27 of
// the ring search, which runs when there is no such vertex or the box is
// larger.  Runs on a second stream while the site KNN runs; k_site_clip is
// the first kernel to read a.nnv.
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_frame_vertex(EngineArgs<T> a, int parity) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= __ldg(a.act_count)) return;
  const int g = a.act[w];
  const MeshDev& md = a.meshes[a.segs[__ldg(a.site_seg + g)].mesh];
  const V3<T> q = ldp(a.S[parity], g);
  auto all = [](uint32_t) { return true; };
  TopK<T, 1> nv;
  const int old = a.nnv[g];
  bool done = false;
  if ((unsigned)old < (unsigned)md.nV) {
    const V3<T> pv{(T)__ldg(md.V + 3 * old), (T)__ldg(md.V + 3 * old + 1), (T)__ldg(md.V + 3 * old + 2)};
    const T thr = dist2(pv, q);
    const float qm = fmaxf(fabsf((float)q.x), fmaxf(fabsf((float)q.y), fabsf((float)q.z)));
    const float rad = __fsqrt_ru(f32_ru(thr)) * 1.0001f + 1e-3f * md.vg.h + 4e-7f * qm;
    done = grid_knn_box<T, float, 1>(md.vg, md.vcell_start, md.vsorted, q, thr, rad, nv, all, kVertexBoxCells);
    if (!done) nv = TopK<T, 1>();
  }
  if (!done) grid_knn<T, float, 1>(md.vg, md.vcell_start, md.vsorted, q, nv, all);
  a.nnv[g] = (int)KeyOps<T>::idx(nv.k[0]);
}

// ---------------------------------------------------------------------------
// Site KNN (k_knn_verify + k_knn_search): exact K nearest other sites
// within the site's segment (the reference's K+1 nearest with self dropped,
// site_knn.cuh:79-103).  Sets same[g] (new list == stored list) and kth[g].
// ---------------------------------------------------------------------------
// Candidate lists (MM > 0): besides its K neighbours, a site keeps the MM
// nearest other sites of its last full search (ids and the MM-th squared
// distance r2b = rho^2) and a bound D on how much closer any other site can
// have come since.  Every iteration adds to D the site's own last motion and
// the largest last motion of any site in the 8 coarse blocks (kBlockCells^3
// cells each, edge B = kBlockCells h) nearest the site's old position, which
// reach at least B/2 beyond it on every side.  A site j outside the list
// started at distance >= rho; while it starts a step within B/2 of site i
// its step is among those counted, and from farther it cannot end the step
// within rho as long as (largest motion of the step in the segment) + (i's
// motion) < B/2 - rho, which every iteration checks.  So when the K-th nearest
// of the re-keyed list is closer than rho - D, no site outside the list is
// closer: the list's first K are exactly the K nearest of all, the keys a
// full search returns, at a fraction of its work.  Otherwise (and in a
// segment's first iteration) the full search runs for MM neighbours and
// refreshes the list.  Margins of 1e-4 cover the rounding of the distances
// and of the accumulated motion; a NaN motion fails every test.

// Full search of site g (one warp): the K nearest (MM = 0), or the MM
// nearest, which refresh its candidate list and whose first K are the
// K-list.  seg receives the site's segment.  With candidate lists the search
// is first tried as one radius query (warp_radius_knn, scratch buf of
// kRadiusKeys keys): within bound tb when the check left one (the largest
// re-keyed distance of the site's complete old list, so at least MM sites lie
// within it), else within a squared distance expected to hold 1.45 MM sites;
// when that fails (too few or too many) the ring search runs instead.  Both
// return the MM smallest (distance, caller index) keys; the list is stored as
// internal indices.
template <class T, int KK, int MM>
__device__ __forceinline__ void knn_search_site(const EngineArgs<T>& a, int parity, int g, float tb, int lane, int& seg,
                                                typename KeyOps<T>::Key* buf) {
  using O = KeyOps<T>;
  using Key = typename O::Key;
  constexpr int LEN = MM > 0 ? MM : KK;  // entries stored
  constexpr int R = (LEN + 31) / 32;
  const Pt4<T> me = a.S[parity][g];
  const int s = __ldg(a.site_seg + g);
  seg = s;
  const SegDev& sd = a.segs[s];
  // The K nearest other sites: the reference's K+1 nearest with self dropped
  // (site_knn.cuh:79-103) are exactly these, also when duplicates of the site
  // with smaller indices push self out of the K+1 (then the first K are kept,
  // the same K points), and the K-th distance equals the (K+1)-th with self.
  const V3<T> q{me.x, me.y, me.z};
  const float kp = a.kth[g];
  const uint32_t self = me.id;
  auto not_self = [self](uint32_t id) { return id != self; };
  Key mk[2] = {O::empty(), O::empty()};
  if constexpr (MM > 0) {
    const float rho = a.cand_rho[g];
    const GridGeom G = a.geom[s];
    // kth holds the site's last K-th squared distance (K sites within it);
    // kth_est, from the segment's density, is expected to hold 2 (K + 1)
    constexpr double kTarget = 1.45 * MM;
    const T thr_r = tb >= 0.f ? (T)tb
                    : kp >= 0.f ? (T)kp * (T)(kTarget / KK) : (T)sd.kth_est * (T)(kTarget / (2.0 * (KK + 1)));
    const float qm = fmaxf(fabsf((float)q.x), fmaxf(fabsf((float)q.y), fabsf((float)q.z)));
    const float rad = __fsqrt_ru(f32_ru(thr_r)) * 1.0001f + 1e-3f * G.h + 4e-7f * qm;
    if (!warp_radius_knn<T, T, MM>(G, a.cell_start, a.sorted, q, thr_r, rad, lane, not_self, buf, mk)) {
      const T thrM = tb >= 0.f ? (T)tb
                     : rho >= 0.f && !isinf(rho) ? (T)rho * (T)rho * (T)1.2
                     : (kp >= 0.f ? (T)kp * (T)(1.1 * (MM + 1) / (KK + 1)) : (T)sd.kth_est * (T)((MM + 1.0) / (KK + 1)));
      if constexpr (MM > 32) {
        warp_knn<T, T, MM>(G, a.cell_start, a.sorted, q, thrM, lane, not_self, mk);
      } else {
        Key one[1];
        warp_knn<T, T, MM>(G, a.cell_start, a.sorted, q, thrM, lane, not_self, one);
        mk[0] = one[0];
        mk[1] = O::empty();
      }
    }
    const Key mth = shfl_key(mk[(MM - 1) / 32], (MM - 1) % 32);
    if (lane == 0) {
      a.cand_rho[g] = O::is_empty(mth) ? __int_as_float(0x7f800000) : __fsqrt_rd(f32_rd(O::dist(mth)));
      a.cand_D[g] = 0.f;
    }
  } else {
    (void)tb; (void)buf;
    // candidates beyond 1.1x the last K-th squared distance are skipped; sites
    // move little between iterations, and a bound that proves too tight
    // restarts the search without it (swept 1.02-1.5: 1.05-1.1 fastest)
    const T thr0 = kp >= 0.f ? (T)kp * (T)1.1 : (T)sd.kth_est;
    Key kl[1];
    warp_knn<T, T, KK>(a.geom[s], a.cell_start, a.sorted, q, thr0, lane, not_self, kl);
    mk[0] = kl[0];
  }
  const Key kth = shfl_key(mk[0], KK - 1);
  uint32_t* col = a.list + (MM > 0 ? (size_t)g : (size_t)g * KK);  // list_site, list_entry
  const size_t step = MM > 0 ? a.stride : 1;
  bool diff = false;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int e = 32 * r + lane;
    if (e < LEN) {
      const uint32_t id = O::idx(mk[r]);
      const uint32_t v = id == 0xffffffffu ? id : __ldg(a.internal_of + id);
      if (e < KK) diff = diff || col[e * step] != v;
      col[e * step] = v;
    }
  }
  const unsigned changed = __ballot_sync(0xffffffffu, diff);
  if (lane == 0) {
    a.kth[g] = O::is_empty(kth) ? -1.f : (float)O::dist(kth);
    a.same[g] = changed ? 0 : 1;
  }
}

// A thread's K (distance, internal index) keys in shared memory: entry t of
// thread c at column c, so that a warp's accesses are conflict-free.
template <class T, int KK, int BS> struct KeyColumns {
  T d[KK][BS];
  uint32_t i[KK][BS];
  __device__ __forceinline__ void get(int t, int c, T& dd, uint32_t& id) const { dd = d[t][c]; id = i[t][c]; }
  __device__ __forceinline__ void put(int t, int c, T dd, uint32_t id) { d[t][c] = dd; i[t][c] = id; }
};
template <int KK, int BS> struct KeyColumns<float, KK, BS> {
  uint2 k[KK][BS];
  __device__ __forceinline__ void get(int t, int c, float& dd, uint32_t& id) const {
    const uint2 v = k[t][c];
    dd = __uint_as_float(v.x); id = v.y;
  }
  __device__ __forceinline__ void put(int t, int c, float dd, uint32_t id) { k[t][c] = make_uint2(__float_as_uint(dd), id); }
};

// Candidate-list check of active site g, one thread.  The motion bound D
// grows by the largest last motion M in the 8 coarse blocks nearest the
// site's old position, which hold every site that started the step within
// B/2 of it, plus the site's own motion; the step condition asks that the
// segment's largest motion plus the site's own stay below B/2 - rho (B/2
// shrunk by 1e-3 for the rounding of cell coordinates), so a site that
// started the step outside those blocks ends it beyond rho.  The list is
// re-keyed at the current positions and its KK smallest kept in order by
// insertion (the head of the list is the order of the last iteration, so most
// entries go straight to the end); an entry pushed out of the first KK takes
// the place of the one that pushed it.  Equal distances compare the caller's
// indices.  The list is accepted when the KK-th is closer than rho - D.  True
// when the K-list came from the list (and is stored: the entries that
// changed, kth, same, D).  bound: for a site whose complete list was
// re-keyed, the largest re-keyed squared distance rounded up (its MM list
// sites are MM other sites, so the MM nearest lie within it); else -1.  A
// rejected list is rewritten by the full search.
template <class T, int KK, int MM, int BS>
__device__ __forceinline__ bool knn_verify_site(const EngineArgs<T>& a, int parity, int g, int s,
                                                KeyColumns<T, KK, BS>& L, float& bound) {
  static_assert(MM > KK && MM % 4 == 0, "four entries per step");
  constexpr uint32_t kNone = 0xffffffffu;
  bound = -1.f;
  const float rho = a.cand_rho[g];
  if (!(rho >= 0.f)) return false;
  const Pt4<T>* __restrict__ S = a.S[parity];
  const int c = threadIdx.x;
  uint32_t* col = a.list + g;
  uint32_t id[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) id[j] = col[j * a.stride];
  const V3<T> q = ldp(S, g);
  float D, lim;
  bool ok;
  {
    const SegDev& sd = a.segs[s];
    const GridGeom& G = a.geom[s];
    // the 2 x 2 x 2 blocks nearest the old position: per axis the block of
    // its cell and the neighbour on the side of the nearer block face, which
    // reach at least kBlockCells / 2 cells beyond the cell on either side
    const V3<T> po = ldp(a.S[parity ^ 1], g);
    const int c0[3] = {grid_coord(G, po.x, 0), grid_coord(G, po.y, 1), grid_coord(G, po.z, 2)};
    int b0[3], nb[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      b0[ax] = c0[ax] / kBlockCells - (c0[ax] % kBlockCells < kBlockCells / 2 ? 1 : 0);
      nb[ax] = block_dim(G, ax);
    }
    const unsigned stamp = (unsigned)(sd.iter - 1);
    unsigned mbits = 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int x = b0[0] + (k & 1), y = b0[1] + ((k >> 1) & 1), z = b0[2] + (k >> 2);
      if (x >= 0 && x < nb[0] && y >= 0 && y < nb[1] && z >= 0 && z < nb[2]) {
        const unsigned long long v = a.blockmax[G.cell_base + (z * nb[1] + y) * nb[0] + x];
        if ((unsigned)(v >> 32) == stamp) mbits = max(mbits, (unsigned)v);
      }
    }
    // this site's own motion (also inside M, but usually far below it)
    const float mu = __fsqrt_rn(f32_ru(dist2(q, po))) * 1.000001f;
    D = __fadd_ru(a.cand_D[g], __fadd_ru(__uint_as_float(mbits), mu));
    const bool step_ok = __fadd_ru(sd.step_motion, mu) * 1.0001f < (0.4995f * (float)kBlockCells * G.h - rho) * 0.9999f;
    lim = rho * 0.9999f - D * 1.0001f;
    ok = isinf(rho) || (step_ok && lim > 0.f);
  }
  auto less = [&](T da, uint32_t ia, T db, uint32_t ib) {
    if (da != db) return da < db;
    return S[ia].id < S[ib].id;
  };
  T dmax = (T)0, dk = (T)0;  // largest distance; the last kept key
  uint32_t ik = kNone;
  int cnt = 0, nv = 0, lo = KK;  // kept keys, list entries, first position that changed
  bool finite = true;
#pragma unroll 1
  for (int e0 = 0; e0 < MM; e0 += 4) {
    uint32_t cur[4];
    V3<T> p[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      cur[j] = id[j];
      p[j] = cur[j] != kNone ? ldp(S, cur[j]) : q;
      if (e0 + 4 < MM) id[j] = col[(e0 + 4 + j) * a.stride];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (cur[j] == kNone) continue;
      const T d = dist2(p[j], q);
      ++nv;
      finite = finite && d < (T)INFINITY;
      dmax = d > dmax ? d : dmax;
      if (!ok) continue;
      const bool below = cnt > 0 && less(d, cur[j], dk, ik);
      if (!below) {
        if (cnt < KK) { L.put(cnt++, c, d, cur[j]); dk = d; ik = cur[j]; }
        continue;
      }
      const bool full = cnt == KK;
      if (full) col[(e0 + j) * a.stride] = ik; else ++cnt;
      int t = cnt - 1;
      while (t > 0) {
        T dt;
        uint32_t it;
        L.get(t - 1, c, dt, it);
        if (!less(d, cur[j], dt, it)) break;
        L.put(t, c, dt, it);
        --t;
      }
      L.put(t, c, d, cur[j]);
      lo = min(lo, t);
      if (full) L.get(KK - 1, c, dk, ik);
    }
  }
  bound = nv == MM && finite ? f32_ru(dmax) : -1.f;
  ok = ok && cnt == KK && finite && (isinf(rho) || f32_ru(dk) * 1.0003f < lim * lim);
  if (ok) {
    for (int t = lo; t < KK; ++t) {
      T dt;
      uint32_t it;
      L.get(t, c, dt, it);
      col[t * a.stride] = it;
    }
    a.cand_D[g] = D;
    a.kth[g] = (float)dk;
    a.same[g] = lo == KK ? 1 : 0;
  }
  return ok;
}

// k_knn_verify: the check of every active site, one thread per site; the
// sites it leaves are appended to a.srch once per block, the lists it proved
// are added to their segment's statistics (word 6 of the iteration's slot).
// Bound by instruction issue and the latency of the gathers.  Measured on 300k
// sites, K = 24, after 10 iterations: 75 us at 116 warp instructions per site;
// a half warp per site with the keys in registers (odd-even passes over
// shuffles, 12-byte positions in the caller's order) took 167 us and 358.
// 64 threads: 12 KB of keys (K = 24), 16 blocks on an SM.
constexpr int kVerifyThreads = 64;

template <class T, int KK, int MM>
__global__ void __launch_bounds__(kVerifyThreads, sizeof(T) == 8 ? 8 : 16) k_knn_verify(EngineArgs<T> a, int parity) {
  constexpr int BS = kVerifyThreads;
  __shared__ KeyColumns<T, KK, BS> L;
  __shared__ int warp_base[BS / 32], block_base, st_seg, st_n;
  const int n = __ldg(a.act_count);
  if (blockIdx.x * BS >= n) return;
  if (threadIdx.x == 0) { st_seg = -1; st_n = 0; }
  const int w = blockIdx.x * BS + threadIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int g = -1, s = -1;
  float bound = -1.f;
  bool ok = false;
  if (w < n) {
    g = a.act[w];
    s = __ldg(a.site_seg + g);
    ok = knn_verify_site<T, KK, MM, BS>(a, parity, g, s, L, bound);
  }
  const bool need = g >= 0 && !ok;
  const unsigned m = __ballot_sync(0xffffffffu, need);
  if (lane == 0) warp_base[wid] = __popc(m);
  __syncthreads();
  const int key = ok ? s : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  if (key >= 0 && lane == __ffs(peers) - 1) {
    const int owner = atomicCAS(&st_seg, -1, key);
    int* word = a.stats + ((size_t)key * kStatsRing + (a.segs[key].iter % kStatsRing)) * kStatsWords + 6;
    if (owner == -1 || owner == key) atomicAdd(&st_n, __popc(peers)); else atomicAdd(word, __popc(peers));
  }
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int k = 0; k < BS / 32; ++k) {
      const int cw = warp_base[k];
      warp_base[k] = sum;
      sum += cw;
    }
    block_base = sum ? atomicAdd(a.srch, sum) : 0;
  }
  __syncthreads();
  if (need) {
    const int slot = block_base + warp_base[wid] + __popc(m & ((1u << lane) - 1u));
    a.srch[1 + slot] = g;
    a.srch_thr[slot] = bound;
  }
  if (threadIdx.x == 0 && st_seg >= 0)
    atomicAdd(a.stats + ((size_t)st_seg * kStatsRing + (a.segs[st_seg].iter % kStatsRing)) * kStatsWords + 6, st_n);
}

// Per-warp running count of one statistics word for the segment it is on:
// added to the segment's slot when the segment changes and at the end.
template <class T>
struct SegCounter {
  int cur = -1, n = 0;
  __device__ __forceinline__ void add(const EngineArgs<T>& a, int seg, int word, int lane) {
    if (seg != cur) { flush(a, word, lane); cur = seg; n = 0; }
    ++n;
  }
  __device__ __forceinline__ void flush(const EngineArgs<T>& a, int word, int lane) {
    if (lane == 0 && cur >= 0 && n)
      atomicAdd(a.stats + ((size_t)cur * kStatsRing + (a.segs[cur].iter % kStatsRing)) * kStatsWords + word, n);
  }
};

// k_knn_search: full searches, persistent with the warps its launch bounds
// keep resident on every SM (so no block waits for a second wave), one warp
// per site: the sites the check left (a.srch), or without candidate lists
// (MM = 0) every active site.  Counted in word 7 of the statistics.
constexpr int kKnnSearchWarpsPerSM = 32;

template <class T, int KK, int MM, int BS>
__global__ void __launch_bounds__(BS, kKnnSearchWarpsPerSM * 32 / BS) k_knn_search(EngineArgs<T> a, int parity) {
  const int lane = threadIdx.x & 31;
  const int wi = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
  const int nw = (int)((gridDim.x * (unsigned)blockDim.x) >> 5);
  SegCounter<T> searched;
  if constexpr (MM > 0) {
    __shared__ typename KeyOps<T>::Key buf[BS / 32][kRadiusKeys];  // per warp: the radius query's keys
    auto* mybuf = buf[threadIdx.x >> 5];
    const int n = a.srch[0];
    for (int k = wi; k < n; k += nw) {
      int seg;
      knn_search_site<T, KK, MM>(a, parity, a.srch[1 + k], a.srch_thr[k], lane, seg, mybuf);
      searched.add(a, seg, 7, lane);
    }
  } else {
    const int n = __ldg(a.act_count);
    for (int w = wi; w < n; w += nw) {
      int seg;
      knn_search_site<T, KK, MM>(a, parity, a.act[w], -1.f, lane, seg, nullptr);
      searched.add(a, seg, 7, lane);
    }
  }
  searched.flush(a, 7, lane);
}

// ---------------------------------------------------------------------------
// per-site step after the KNN
// ---------------------------------------------------------------------------
struct SiteOut {
  int seg;
  int same, low, both, newly;
  float disp2;
};

// Frame, clip and centroid of site g into a.cent; false when clip_cell gave
// the cell back (the site is then redone by k_clip_overflow: FULL, with a
// second buffer B).
template <int PROF, int FRAME, bool FULL>
__device__ __forceinline__ bool site_clip(const EngineArgs<typename PT<PROF>::T>& a, int parity, int g,
                                          PolyRef<typename PT<PROF>::PP> A, PolyRef<typename PT<PROF>::PP> B,
                                          int cap) {
  using T = typename PT<PROF>::T;
  using PP = typename PT<PROF>::PP;
  const int s = __ldg(a.site_seg + g);
  const SegDev& sd = a.segs[s];
  const MeshDev& md = a.meshes[sd.mesh];
  const ListNeighbours<T> nb{a.S[parity], a.list + g * a.list_site, a.list_entry};
  const bool fz = sd.mode != 0 && a.frozen[g];
  const V3<T> si = ldp(a.S[parity], g);
  // frame from the nearest vertex normal (frozen sites: their kept vertex
  // list; with the BVH projection, which keeps no vertex list, their kept
  // frame vertex); FRAME 1: from the PCA normal of the neighbour list,
  // started from that vertex normal
  const int nn = (fz && a.proj_mode == 0) ? a.knnv[g] : a.nnv[g];
  Frame<T> fr;
  if (nn < 0) {
    fr = {{(T)1, (T)0, (T)0}, {(T)0, (T)1, (T)0}};
  } else {
    V3<T> n0{(T)__ldg(md.N + 3 * nn), (T)__ldg(md.N + 3 * nn + 1), (T)__ldg(md.N + 3 * nn + 2)};
    if (FRAME == 1) n0 = pca_normal<T>(nb, a.K, si, n0);
    fr = frame_from_normal(n0);
  }
  PolyRef<PP> cur = A, nxt = B;
  const int np = FULL ? clip_cell_full<PROF>(nb, si, a.K, fr, md.R, cur, nxt, cap, !fz)
                      : clip_cell<PROF>(nb, si, a.K, fr, 1.f, md.R, A, cap, !fz);
  if (np < 0) return false;
  const V2<PP> c2 = poly_centroid<PP>(cur, np, PROF == PROF_MIXED);
  V3<T> cent;
  if (!(finiteT(c2.x) && finiteT(c2.y))) {
    cent = {(T)NAN, (T)NAN, (T)NAN};
  } else {
    const T cx = (T)c2.x, cy = (T)c2.y;
    cent = {si.x + fmaT(fr.u.x, cx, fr.v.x * cy), si.y + fmaT(fr.u.y, cx, fr.v.y * cy),
            si.z + fmaT(fr.u.z, cx, fr.v.z * cy)};
  }
  st3(a.cent, g, cent);
  return true;
}

template <int PROF, int BLOCK, int CAP, int FRAME>
__global__ void __launch_bounds__(BLOCK, (sizeof(typename PT<PROF>::PP) == 8 ? kClipThreadsD : kClipThreadsF) / BLOCK)
    k_site_clip(EngineArgs<typename PT<PROF>::T> a, int parity) {
  using PP = typename PT<PROF>::PP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V2<PP>* sm = reinterpret_cast<V2<PP>*>(smem_raw);
  const PolyRef<PP> A{sm + threadIdx.x, BLOCK};
  const int g = blockIdx.x * BLOCK + threadIdx.x;
  if (active_seg(a, g) >= 0) {
    if (!site_clip<PROF, FRAME, false>(a, parity, g, A, A, CAP)) {
      const int k = atomicAdd(a.ovf, 1);
      a.ovf[1 + k] = g;
    }
  }
}

template <int PROF, int FRAME>
__global__ void __launch_bounds__(64) k_clip_overflow(EngineArgs<typename PT<PROF>::T> a, int parity) {
  using PP = typename PT<PROF>::PP;
  V2<PP> buf[2][kFallbackCap];
  const int n = *(volatile int*)a.ovf;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    site_clip<PROF, FRAME, true>(a, parity, a.ovf[1 + k], PolyRef<PP>{buf[0], 1}, PolyRef<PP>{buf[1], 1}, kFallbackCap);
}

// The new position sn of site g, tiers and the freeze test.
template <int PROF>
__device__ __forceinline__ void site_settle(const EngineArgs<typename PT<PROF>::T>& a, int parity, int g,
                                            V3<typename PT<PROF>::T> sn, SiteOut& o);

// Projection, tiers and the freeze test of site g, given the centroid in
// a.cent and (PROJ 0) its 5 nearest vertices knnv; PROJ 1 projects through
// the mesh's BVH and ignores knnv.
template <int PROF, int PROJ, int BS>
__device__ __forceinline__ void site_finish(const EngineArgs<typename PT<PROF>::T>& a, int parity, int g,
                                            const int (&knnv)[kKProj], RingList<BS>& L, SiteOut& o) {
  using T = typename PT<PROF>::T;
  using Q = typename PT<PROF>::Q;
  const int s = __ldg(a.site_seg + g);
  const SegDev& sd = a.segs[s];
  const MeshDev& md = a.meshes[sd.mesh];
  const V3<T> si = ldp(a.S[parity], g);
  const V3<T> cent = ld3((const T*)a.cent, g);

  // projection
  V3<T> sn;
  if (PROF == PROF_MIXED && !finite3(cent)) {
    sn = si;
  } else if (PROJ == 1) {
    sn = project_bvh<T, Q>(cent, md.bvh, (Q)bvh_bound2(cent, si), a.bvh_ovf);
  } else if (!project_onering_rec<T, Q, BS>(cent, md.ring_head, md.ring_body, md.nV, md.vf_off, knnv, L, sn)) {
    sn = project_onering_plain<T, Q>(cent, md.V, md.nV, md.F, md.nF, md.vf_off, md.vf_faces, knnv, kKProj);
  }
  site_settle<PROF>(a, parity, g, sn, o);
}

template <int PROF>
__device__ __forceinline__ void site_settle(const EngineArgs<typename PT<PROF>::T>& a, int parity, int g,
                                            V3<typename PT<PROF>::T> sn, SiteOut& o) {
  using T = typename PT<PROF>::T;
  const int s = __ldg(a.site_seg + g);
  const SegDev& sd = a.segs[s];
  const MeshDev& md = a.meshes[sd.mesh];
  const bool fz = sd.mode != 0 && a.frozen[g];
  const Pt4<T> me = a.S[parity][g];
  const V3<T> si{me.x, me.y, me.z};
  a.S[parity ^ 1][g] = Pt4<T>{sn.x, sn.y, sn.z, me.id};

  // tiers on the segment's first iteration (modes 1/2)
  const int it = sd.iter;
  if (it == 0 && sd.mode != 0) {
    auto normal = [&](int j, float out[3]) {
      int v = a.nnv[j];
      if (v < 0) { out[0] = out[1] = out[2] = 0.f; return; }
      out[0] = __ldg(md.N + 3 * v); out[1] = __ldg(md.N + 3 * v + 1); out[2] = __ldg(md.N + 3 * v + 2);
    };
    auto row = [&](int t) { return (int)a.list[g * a.list_site + t * a.list_entry]; };
    a.tier[g] = (uint8_t)tier_of(sd.mode, g, a.K, row, normal);
  }

  // freeze test + apply
  o.seg = s;
  o.same = o.low = o.both = o.newly = 0;
  const T d2 = dist2(sn, si);
  o.disp2 = (float)d2;
  if (it == 0) {
    a.streak[g] = 0;
  } else {
    const int tt = min((int)a.tier[g], 5);
    // a frozen site's list is the previous one by construction
    const bool same = fz || a.same[g] != 0;
    const bool low = d2 <= (T)sd.thr2_tier[tt];
    const bool both = same && low;
    int st = a.streak[g];
    st = both ? (st < 255 ? st + 1 : st) : 0;
    const bool cand = st >= sd.need_tier[tt];
    o.same = same; o.low = low; o.both = both;
    if (sd.mode == 0) {
      a.streak[g] = 0;   // mode 0 clears streak and frozen every iteration (main.cu:837-846)
    } else {
      a.streak[g] = (uint8_t)st;
      if (cand && !a.frozen[g]) { a.frozen[g] = 1; o.newly = 1; }
    }
  }
}

// Rings the per-thread centroid -> vertex search may visit before the site
// is handed to k_site_far (a centroid far off the surface, e.g. of a cell
// that the neighbours leave almost unbounded in the first iteration).
constexpr int kVertexRingLimit = 4;

// Centroid -> its kKProj nearest mesh vertices, for every gridded site that
// is not frozen (one thread per site), into a.knnv.  A site whose search
// would pass kVertexRingLimit rings is listed in a.far and its list marked
// kVertexDeferred; k_site_far finishes it.  A kernel of its own: the search
// needs a fraction of the projection's registers, so it runs at twice the
// projection's resident warps (FP32 positions: 48 per SM, measured 3 %
// faster for the projection group than the compiler's 56 registers and no
// faster at 64; FP64 positions keep the compiler's choice, which spills
// less).
constexpr int kVertexDeferred = -2;

template <int PROF, int BS>
__global__ void __launch_bounds__(BS, PROF == PROF_FP64 ? 1 : 1536 / BS) k_site_vsearch(EngineArgs<typename PT<PROF>::T> a, int parity) {
  using T = typename PT<PROF>::T;
  const int g = blockIdx.x * BS + threadIdx.x;
  const int s = active_seg(a, g);
  if (s < 0) return;
  const SegDev& sd = a.segs[s];
  if (sd.mode != 0 && a.frozen[g]) return;  // frozen sites keep their vertices
  const MeshDev& md = a.meshes[sd.mesh];
  int* kv = a.knnv + g;
  const int skip = (sd.mode == 0 && sd.ex_quirk) ? (int)a.S[parity][g].id - sd.site_base : -1;
  auto accept = [skip](uint32_t id) { return (int)id != skip; };
  const V3<T> c = ld3((const T*)a.cent, g);
  TopK<T, kKProj> top;
  // the site's 5 vertices of the last iteration lie within the largest of
  // their squared distances to the new centroid, so the 5 nearest do: one
  // box query of the cells within it (exact when it finds 5 vertices)
  bool done = false;
  {
    T thr = (T)0;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < kKProj; ++k) {
      const int v = kv[k * a.stride];
      ok = ok && (unsigned)v < (unsigned)md.nV && v != skip;
      if (ok) {
        const V3<T> pv{(T)__ldg(md.V + 3 * v), (T)__ldg(md.V + 3 * v + 1), (T)__ldg(md.V + 3 * v + 2)};
        const T d = dist2(pv, c);
        thr = d > thr ? d : thr;
      }
    }
    if (ok) {
      const float qm = fmaxf(fabsf((float)c.x), fmaxf(fabsf((float)c.y), fabsf((float)c.z)));
      const float rad = __fsqrt_ru(f32_ru(thr)) * 1.0001f + 1e-3f * md.vg.h + 4e-7f * qm;
      done = grid_knn_box<T, float, kKProj>(md.vg, md.vcell_start, md.vsorted, c, thr, rad, top, accept,
                                            kVertexBoxCells);
      if (!done) top = TopK<T, kKProj>();
    }
  }
  if (!done && !grid_knn<T, float, kKProj>(md.vg, md.vcell_start, md.vsorted, c, top, accept, kVertexRingLimit)) {
    const int k = atomicAdd(a.far, 1);
    a.far[1 + k] = g;
    kv[0] = kVertexDeferred;
    return;
  }
#pragma unroll
  for (int k = 0; k < kKProj; ++k) kv[k * a.stride] = (int)KeyOps<T>::idx(top.k[k]);
}

// Few sites (a.n_sites <= kFewSites[profile]): the vertex search and the
// projection with 8 lanes per site each, which shorten a site's chain of loads
// where one thread each would leave most of the chip idle.  The same results:
// the lanes' candidates are merged by the keys that one thread compares.
// Iteration of a lone segment on a 40k-face torus, K = 20, lanes / threads (us):
// ref 2k sites 62 / 94, 16k 72 / 85, 32k 86 / 88, 40k 95 / 88; mixed 16k 83 / 92,
// 24k 93 / 93, 28k 96 / 94, 40k 108 / 95; fp64 16k 83 / 93, 20k 89 / 94, 24k
// 98 / 95, 32k 102 / 96 (K = 12 and 32 cross at the same places).  16 lanes for
// the projection: 60 at 2k, 75 at 16k; 4 for the search: 79 at 2k.
constexpr int kFewSites[3] = {32768, 25000, 22000};
constexpr int kVsearchLanes = 8;
constexpr int kProjLanes = 8;

template <int PROF>
__global__ void __launch_bounds__(128) k_site_vsearch_lanes(EngineArgs<typename PT<PROF>::T> a, int parity) {
  using T = typename PT<PROF>::T;
  using O = KeyOps<T>;
  using Key = typename O::Key;
  constexpr unsigned full = 0xffffffffu;
  const int g = (int)(blockIdx.x * 128u + threadIdx.x) / kVsearchLanes;
  const int sub = threadIdx.x & (kVsearchLanes - 1);
  const int s = active_seg(a, g);
  const bool in = s >= 0 && !(a.segs[s].mode != 0 && a.frozen[g]);  // frozen sites keep their vertices
  const MeshDev& md = a.meshes[in ? a.segs[s].mesh : 0];
  int skip = -1;
  V3<T> c{0, 0, 0};
  T thr = (T)0;
  bool ok = false;
  if (in) {
    const SegDev& sd = a.segs[s];
    skip = (sd.mode == 0 && sd.ex_quirk) ? (int)a.S[parity][g].id - sd.site_base : -1;
    c = ld3((const T*)a.cent, g);
    ok = true;
    if (sub < kKProj) {
      const int v = a.knnv[sub * a.stride + g];
      ok = (unsigned)v < (unsigned)md.nV && v != skip;
      if (ok) thr = dist2(V3<T>{(T)__ldg(md.V + 3 * v), (T)__ldg(md.V + 3 * v + 1), (T)__ldg(md.V + 3 * v + 2)}, c);
    }
  }
  // the box of k_site_vsearch: within the largest of the five distances
#pragma unroll
  for (int o = kVsearchLanes / 2; o > 0; o >>= 1) {
    const T x = __shfl_xor_sync(full, thr, o);
    thr = x > thr ? x : thr;
  }
  const unsigned group = ((1u << kVsearchLanes) - 1u) << (threadIdx.x & 31 & ~(kVsearchLanes - 1));
  bool box = (__ballot_sync(full, ok) & group) == group && finite3(c) && thr >= (T)0;
  TopK<T, kKProj> top;
  if (box) {
    const GridGeom& G = md.vg;
    const float qf[3] = {(float)c.x, (float)c.y, (float)c.z};
    const float qm = fmaxf(fabsf(qf[0]), fmaxf(fabsf(qf[1]), fabsf(qf[2])));
    const float rad = __fsqrt_ru(f32_ru(thr)) * 1.0001f + 1e-3f * G.h + 4e-7f * qm;
    int lo[3], hi[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      lo[ax] = grid_coord(G, __fsub_rd(qf[ax], rad), ax);
      hi[ax] = grid_coord(G, __fadd_ru(qf[ax], rad), ax);
    }
    const int ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1;
    box = rad < INFINITY && (hi[0] - lo[0] + 1) * ny * nz <= kVertexBoxCells;
    if (box)
      for (int r = sub; r < ny * nz; r += kVsearchLanes) {
        const int row = G.cell_base + ((lo[2] + r / ny) * G.dim[1] + lo[1] + r % ny) * G.dim[0];
        const int e = __ldg(md.vcell_start + row + hi[0] + 1);
        for (int k = __ldg(md.vcell_start + row + lo[0]); k < e; ++k) {
          const Pt4<float> p = md.vsorted[k];
          if ((int)p.id == skip) continue;
          const T d = dist2(V3<T>{(T)p.x, (T)p.y, (T)p.z}, c);
          if (d <= thr && d <= top.worst_d()) top.insert(O::make(d, p.id));
        }
      }
  }
  // the group's five smallest keys, smallest first; the lane that holds one
  // moves on to its next
  Key out[kKProj];
#pragma unroll
  for (int k = 0; k < kKProj; ++k) {
    Key m = top.k[0];
#pragma unroll
    for (int o = kVsearchLanes / 2; o > 0; o >>= 1) m = O::kmin(m, shfl_xor_key(m, o));
    out[k] = m;
    if (!O::less(m, top.k[0])) {
#pragma unroll
      for (int j = 0; j + 1 < kKProj; ++j) top.k[j] = top.k[j + 1];
      top.k[kKProj - 1] = O::empty();
    }
  }
  if (!in) return;
  if (!(box && !O::is_empty(out[kKProj - 1]))) {
    if (sub != 0) return;
    top = TopK<T, kKProj>();
    if (!grid_knn<T, float, kKProj>(md.vg, md.vcell_start, md.vsorted, c, top,
                                    [skip](uint32_t id) { return (int)id != skip; }, kVertexRingLimit)) {
      a.far[1 + atomicAdd(a.far, 1)] = g;
      a.knnv[g] = kVertexDeferred;
      return;
    }
#pragma unroll
    for (int k = 0; k < kKProj; ++k) a.knnv[k * a.stride + g] = (int)O::idx(top.k[k]);
    return;
  }
#pragma unroll
  for (int k = 0; k < kKProj; ++k)
    if (sub == k) a.knnv[k * a.stride + g] = (int)O::idx(out[k]);
}

// Everything after the centroid and (PROJ 0) the vertex search of
// k_site_vsearch; false when that search was deferred (the site is then
// listed in a.far and finished by k_site_far).
template <int PROF, int PROJ, int BS>
__device__ __forceinline__ bool site_proj(const EngineArgs<typename PT<PROF>::T>& a, int parity, int g, RingList<BS>& L,
                                          SiteOut& o) {
  if (PROJ == 1) {
    const int none[kKProj] = {-1, -1, -1, -1, -1};
    site_finish<PROF, 1>(a, parity, g, none, L, o);
    return true;
  }
  int knnv[kKProj];
#pragma unroll
  for (int k = 0; k < kKProj; ++k) knnv[k] = a.knnv[k * a.stride + g];
  if (knnv[0] == kVertexDeferred) return false;
  site_finish<PROF, 0>(a, parity, g, knnv, L, o);
  return true;
}

__device__ __forceinline__ void stats_atomic(int* stats, const SegDev* segs, const SiteOut& o) {
  int* sl = stats + ((size_t)o.seg * kStatsRing + (segs[o.seg].iter % kStatsRing)) * kStatsWords;
  if (o.same) atomicAdd(sl + 0, 1);
  if (o.low) atomicAdd(sl + 1, 1);
  if (o.both) atomicAdd(sl + 2, 1);
  if (o.newly) atomicAdd(sl + 3, 1);
  atomicMax(reinterpret_cast<unsigned*>(sl + 4), __float_as_uint(o.disp2));
}

// Per-block staging of the per-segment counters: the first segment a warp
// of the block reports claims the slot; counts of other segments go to
// global memory directly.  (One set of global atomics per block instead of
// per warp: thousands of warps adding to the same few words serialised in
// L2.)  Sums and a max of float bits, so the totals do not depend on order.
struct StatsStage {
  int seg;
  unsigned v[5];  // same, low, both, newly, max squared displacement (float bits)
};

__device__ __forceinline__ void stats_stage_init(StatsStage& s) {
  if (threadIdx.x < 5) s.v[threadIdx.x] = 0u;
  if (threadIdx.x == 0) s.seg = -1;
}

__device__ __forceinline__ void stats_flush(int* stats, const SegDev* segs, const SiteOut& o, StatsStage& stage) {
  // warp-aggregated per-segment counters; every lane of the warp takes part
  const unsigned full = 0xffffffffu;
  const int key = o.seg;
  const unsigned peers = __match_any_sync(full, key);
  const int leader = __ffs(peers) - 1;
  const int lane = threadIdx.x & 31;
  const int same = __popc(__ballot_sync(full, o.same) & peers);
  const int low = __popc(__ballot_sync(full, o.low) & peers);
  const int both = __popc(__ballot_sync(full, o.both) & peers);
  const int newly = __popc(__ballot_sync(full, o.newly) & peers);
  const unsigned dbits = __reduce_max_sync(peers, __float_as_uint(o.seg >= 0 ? o.disp2 : 0.f));
  if (lane == leader && key >= 0) {
    const int owner = atomicCAS(&stage.seg, -1, key);
    if (owner == -1 || owner == key) {
      if (same) atomicAdd(&stage.v[0], (unsigned)same);
      if (low) atomicAdd(&stage.v[1], (unsigned)low);
      if (both) atomicAdd(&stage.v[2], (unsigned)both);
      if (newly) atomicAdd(&stage.v[3], (unsigned)newly);
      atomicMax(&stage.v[4], dbits);
    } else {
      int* sl = stats + ((size_t)key * kStatsRing + (segs[key].iter % kStatsRing)) * kStatsWords;
      if (same) atomicAdd(sl + 0, same);
      if (low) atomicAdd(sl + 1, low);
      if (both) atomicAdd(sl + 2, both);
      if (newly) atomicAdd(sl + 3, newly);
      atomicMax(reinterpret_cast<unsigned*>(sl + 4), dbits);
    }
  }
}

// after a __syncthreads that follows every warp's stats_flush
__device__ __forceinline__ void stats_stage_flush(int* stats, const SegDev* segs, const StatsStage& stage) {
  if (threadIdx.x != 0 || stage.seg < 0) return;
  int* sl = stats + ((size_t)stage.seg * kStatsRing + (segs[stage.seg].iter % kStatsRing)) * kStatsWords;
  for (int w = 0; w < 4; ++w)
    if (stage.v[w]) atomicAdd(sl + w, (int)stage.v[w]);
  atomicMax(reinterpret_cast<unsigned*>(sl + 4), stage.v[4]);
}

// This step's motion of site g (o from site_finish; o.seg < 0: none) into
// its coarse block at its old position, for the next iteration's KNN:
// warp-collective, one atomic per distinct block of the warp.  The stamp is
// the segment's iteration, so an entry from an earlier iteration reads as
// no motion.
template <class T>
__device__ __forceinline__ void motion_to_block(const EngineArgs<T>& a, int parity, int g, const SiteOut& o) {
  int blk = -1;
  unsigned bits = 0u, stamp = 0u;
  if (g >= 0 && o.seg >= 0) {
    int bx, by, bz;
    blk = motion_block(a.geom[o.seg], ldp(a.S[parity], g), bx, by, bz);
    bits = __float_as_uint(sqrtf(o.disp2));
    stamp = (unsigned)a.segs[o.seg].iter;
  }
  const unsigned peers = __match_any_sync(0xffffffffu, blk);
  const unsigned mb = __reduce_max_sync(peers, bits);
  if (blk >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
    atomicMax(a.blockmax + blk, ((unsigned long long)stamp << 32) | mb);
}

// One-ring projection: 24 resident warps per SM (80 registers); with 32 (64
// registers, spills) it takes the same time.  The BVH projection keeps the
// compiler's choice.
template <int PROF, int BS, int PROJ>
__global__ void __launch_bounds__(BS, PROJ == 0 ? 768 / BS : 1) k_site_proj(EngineArgs<typename PT<PROF>::T> a, int parity) {
  __shared__ StatsStage stage;
  __shared__ RingList<PROJ == 0 ? BS : 1> rings;
  stats_stage_init(stage);
  __syncthreads();
  const int g = blockIdx.x * BS + threadIdx.x;
  SiteOut o{-1, 0, 0, 0, 0, 0.f};
  if (active_seg(a, g) >= 0) site_proj<PROF, PROJ>(a, parity, g, rings, o);
  if (a.blockmax) motion_to_block(a, parity, g, o);
  stats_flush(a.stats, a.segs, o, stage);
  __syncthreads();
  stats_stage_flush(a.stats, a.segs, stage);
}

// k_site_proj (one-ring) with kProjLanes lanes per site; the first lane of a
// site does what follows its projection.
template <int PROF>
__global__ void __launch_bounds__(128) k_site_proj_lanes(EngineArgs<typename PT<PROF>::T> a, int parity) {
  using T = typename PT<PROF>::T;
  using Q = typename PT<PROF>::Q;
  __shared__ StatsStage stage;
  stats_stage_init(stage);
  __syncthreads();
  const int g = (int)(blockIdx.x * 128u + threadIdx.x) / kProjLanes;
  const int s = active_seg(a, g);
  const MeshDev& md = a.meshes[s >= 0 ? a.segs[s].mesh : 0];
  int knnv[kKProj] = {-1, -1, -1, -1, -1};
  V3<T> cent{0, 0, 0};
  bool in = s >= 0;
  if (in) {
#pragma unroll
    for (int k = 0; k < kKProj; ++k) knnv[k] = a.knnv[k * a.stride + g];
    in = knnv[0] != kVertexDeferred;
    cent = ld3((const T*)a.cent, g);
    if (!in || (PROF == PROF_MIXED && !finite3(cent)))
#pragma unroll
      for (int k = 0; k < kKProj; ++k) knnv[k] = -1;
  }
  V3<T> sn = project_onering_lanes<T, Q, kProjLanes>(cent, md.ring_head, md.ring_body, md.nV, md.vf_off, knnv);
  SiteOut o{-1, 0, 0, 0, 0, 0.f};
  const bool lead = in && (threadIdx.x & (kProjLanes - 1)) == 0;
  if (lead) {
    if (PROF == PROF_MIXED && !finite3(cent)) sn = ldp(a.S[parity], g);
    site_settle<PROF>(a, parity, g, sn, o);
  }
  if (a.blockmax) motion_to_block(a, parity, lead ? g : -1, o);
  stats_flush(a.stats, a.segs, o, stage);
  __syncthreads();
  stats_stage_flush(a.stats, a.segs, stage);
}

// Iteration bookkeeping, run by one block: advance active segments, clear
// their next stats slot, apply each segment's stop rule (a stopped segment is
// no longer gridded or iterated: active = 2), reset the overflow, deferred
// and active-site counts for the next iteration.
__device__ __forceinline__ void seg_advance(SegDev* segs, int* active, int nseg, int* stats, int* ovf, int* far,
                                            int* act_count, int* srch) {
  for (int s = threadIdx.x; s < nseg; s += blockDim.x) {
    if (active[s] != 1) continue;
    int it = segs[s].iter;
    int* cur = stats + ((size_t)s * kStatsRing + (it % kStatsRing)) * kStatsWords;
    cur[5] = it;
    const float d2 = __uint_as_float((unsigned)cur[4]);
    int nx = it + 1;
    int* sl = stats + ((size_t)s * kStatsRing + (nx % kStatsRing)) * kStatsWords;
    for (int w = 0; w < kStatsWords; ++w) sl[w] = 0;
    segs[s].iter = nx;
    // the step bound of the candidate lists (NaN fails every test)
    segs[s].step_motion = sqrtf(d2);
    const float lim = segs[s].stop_motion2;
    const int cap = segs[s].stop_iters;
    if ((lim >= 0.f && d2 <= lim) || (cap > 0 && nx >= cap)) active[s] = 2;
  }
  if (threadIdx.x == 0) {
    ovf[0] = 0; far[0] = 0; *act_count = 0;
    if (srch) srch[0] = 0;
  }
}

// Deferred sites (a.far): one block per site finds the 5 nearest mesh
// vertices of the centroid by scanning all of them (each thread every
// kFarThreads-th vertex; exact, the keys are unique), then thread 0 finishes
// the site.  A warp's lists are merged by taking the smallest head five times,
// thread 0 merges the warps'.  With short lists (K = 8) some cells stay open
// and every iteration has such sites: 15.5k sites, K = 8, 70 iterations took
// 12.7 ms with 128 threads and thread 0 merging all 640 keys, 10.7 ms so.
// The last block to finish then runs the iteration's bookkeeping
// (seg_advance), counted by `ticket`, which it leaves at zero.
constexpr int kFarThreads = 256;

template <int PROF>
__global__ void __launch_bounds__(kFarThreads) k_site_far(EngineArgs<typename PT<PROF>::T> a, int parity, SegDev* segs,
                                                   int* active, int nseg, unsigned* ticket) {
  using T = typename PT<PROF>::T;
  using Key = typename KeyOps<T>::Key;
  using O = KeyOps<T>;
  __shared__ Key keys[kFarThreads / 32 * kKProj];
  __shared__ RingList<1> rings;  // thread 0's
  __shared__ bool last;
  const int n = *(volatile int*)a.far;
  for (int k = blockIdx.x; k < n; k += gridDim.x) {
    const int g = a.far[1 + k];
    const int s = __ldg(a.site_seg + g);
    const SegDev& sd = a.segs[s];
    const MeshDev& md = a.meshes[sd.mesh];
    const int skip = (sd.mode == 0 && sd.ex_quirk) ? (int)a.S[parity][g].id - sd.site_base : -1;
    const V3<T> q = ld3((const T*)a.cent, g);
    TopK<T, kKProj> top;
    for (int v = threadIdx.x; v < md.nV; v += kFarThreads) {
      if (v == skip) continue;
      const V3<T> p{(T)__ldg(md.V + 3 * v), (T)__ldg(md.V + 3 * v + 1), (T)__ldg(md.V + 3 * v + 2)};
      const T d = dist2(p, q);
      if (d <= top.worst_d()) top.insert(KeyOps<T>::make(d, (uint32_t)v));
    }
#pragma unroll
    for (int j = 0; j < kKProj; ++j) {
      Key m = top.k[0];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = O::kmin(m, shfl_xor_key(m, o));
      if ((threadIdx.x & 31) == 0) keys[(threadIdx.x >> 5) * kKProj + j] = m;
      if (!O::less(m, top.k[0])) {
#pragma unroll
        for (int q2 = 0; q2 + 1 < kKProj; ++q2) top.k[q2] = top.k[q2 + 1];
        top.k[kKProj - 1] = O::empty();
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      TopK<T, kKProj> all;
      for (int j = 0; j < kFarThreads / 32 * kKProj; ++j) all.insert(keys[j]);
      int knnv[kKProj];
#pragma unroll
      for (int j = 0; j < kKProj; ++j) {
        knnv[j] = (int)KeyOps<T>::idx(all.k[j]);
        a.knnv[j * a.stride + g] = knnv[j];
      }
      SiteOut o{-1, 0, 0, 0, 0, 0.f};
      site_finish<PROF, 0>(a, parity, g, knnv, rings, o);
      stats_atomic(a.stats, a.segs, o);
      if (a.blockmax) {
        int bx, by, bz;
        const int blk = motion_block(a.geom[o.seg], ldp(a.S[parity], g), bx, by, bz);
        atomicMax(a.blockmax + blk, ((unsigned long long)(unsigned)a.segs[o.seg].iter << 32) |
                                        __float_as_uint(sqrtf(o.disp2)));
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  seg_advance(segs, active, nseg, a.stats, a.ovf, a.far, a.act_count, a.srch);
  if (threadIdx.x == 0) *ticket = 0u;
}

}  // namespace cvt
