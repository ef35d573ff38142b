// Mesh ingest on the device: validation, vertex compaction (main.cu:230-257),
// vertex->face CSR in face order (main.cu:259-285), surface area, the
// sampler's face-area prefix sums and the evaluation BVH (evaluate.cuh:114-201).
//
// The BVH is built level by level.  Every node of the reference's recursive
// builder splits its triangles, stably sorted along the longest axis of
// their centroid extent, at the middle.  The tree's shape therefore depends
// on the triangle count only, so the host plans every level (segments of the
// id array, pre-order node numbers) and the device does the data work: per
// segment bounds and centroid extent (warp-aggregated atomics), then one
// stable radix sort of (segment rank, centroid key) pairs over the whole id
// array.  A stable LSD radix sort orders equal keys by their current
// position, exactly as std::stable_sort does, so nodes and triangle order are
// identical to the recursive build.
#pragma once
#include "cvt_eval.cuh"

namespace cvt {

// float -> int whose signed order is the float order (-0 below +0)
__device__ __forceinline__ int ing_f2ord(float v) {
  int b = __float_as_int(v);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float ing_ord2f(int o) { return __int_as_float(o >= 0 ? o : o ^ 0x7fffffff); }

// Face corners: range check (bad |= 1) and referenced-vertex marks.
__global__ void k_ingest_mark(const int* __restrict__ F, long n3, int nV, int* __restrict__ used, int* bad) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n3) return;
  const int v = F[k];
  if ((unsigned)v >= (unsigned)nV) { atomicOr(bad, 1); return; }
  used[v] = 1;
}

// Bounds of every input vertex (R, main.cu:169-227) and of the referenced ones
// (bbox of the compacted mesh); a referenced vertex with a non-finite
// coordinate sets bad |= 2.  bb: all lo[3] hi[3], used lo[3] hi[3] (ord ints).
// Grid-stride blocks with one set of atomics each (a set per warp serialised on
// the twelve words: 26 us for 100k vertices, now 5).
__global__ void __launch_bounds__(256) k_ingest_bounds(const float* __restrict__ V, int nV, const int* __restrict__ used,
                                                       int* bb, int* bad) {
  __shared__ int sb[12];
  if (threadIdx.x < 12) sb[threadIdx.x] = (threadIdx.x % 6) < 3 ? INT_MAX : INT_MIN;
  __syncthreads();
  int lo[6], hi[6];  // all vertices, used vertices
#pragma unroll
  for (int k = 0; k < 6; ++k) { lo[k] = INT_MAX; hi[k] = INT_MIN; }
  for (int i = blockIdx.x * 256 + threadIdx.x; i < nV; i += gridDim.x * 256) {
    const V3<float> p = ld3(V, i);
    const bool u = used[i] != 0;
    if (!finite3(p)) {
      if (u) atomicOr(bad, 2);
      continue;
    }
    const int o[3] = {ing_f2ord(p.x), ing_f2ord(p.y), ing_f2ord(p.z)};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = min(lo[a], o[a]); hi[a] = max(hi[a], o[a]);
      if (u) { lo[3 + a] = min(lo[3 + a], o[a]); hi[3 + a] = max(hi[3 + a], o[a]); }
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int mn = __reduce_min_sync(0xffffffffu, lo[k]), mx = __reduce_max_sync(0xffffffffu, hi[k]);
    if ((threadIdx.x & 31) == 0) { atomicMin(sb + 6 * (k / 3) + k % 3, mn); atomicMax(sb + 6 * (k / 3) + 3 + k % 3, mx); }
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int v = sb[threadIdx.x];
    if ((threadIdx.x % 6) < 3) { if (v != INT_MAX) atomicMin(bb + threadIdx.x, v); }
    else if (v != INT_MIN) atomicMax(bb + threadIdx.x, v);
  }
}

__global__ void k_ingest_bounds_init(int* bb) {
  if (threadIdx.x < 12) bb[threadIdx.x] = (threadIdx.x % 6) < 3 ? INT_MAX : INT_MIN;
}

// Area of each face in FP64, the arithmetic of the host loop (main.cu area
// for the grid density; sampler CDF).
__global__ void k_face_area(const float* __restrict__ V, const int* __restrict__ F, int nF, double* __restrict__ out) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nF) return;
  const float* a = V + 3 * (size_t)F[3 * f];
  const float* b = V + 3 * (size_t)F[3 * f + 1];
  const float* c = V + 3 * (size_t)F[3 * f + 2];
  const double e1x = (double)b[0] - a[0], e1y = (double)b[1] - a[1], e1z = (double)b[2] - a[2];
  const double e2x = (double)c[0] - a[0], e2y = (double)c[1] - a[1], e2z = (double)c[2] - a[2];
  const double cx = e1y * e2z - e1z * e2y, cy = e1z * e2x - e1x * e2z, cz = e1x * e2y - e1y * e2x;
  out[f] = 0.5 * __dsqrt_rn(cx * cx + cy * cy + cz * cz);
}

// used vertex i -> dV[remap[i]]; unused -> dunref[i - remap[i]] (input order)
__global__ void k_ingest_compact(const float* __restrict__ V, int nV, const int* __restrict__ used,
                                 const int* __restrict__ remap, float* __restrict__ dV, float* __restrict__ dunref) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nV) return;
  float* o = used[i] ? dV + 3 * (size_t)remap[i] : dunref + 3 * (size_t)(i - remap[i]);
  o[0] = V[3 * i]; o[1] = V[3 * i + 1]; o[2] = V[3 * i + 2];
}

// faces through the remap; CSR sort keys (vertex << 32 | face) and counts
__global__ void k_ingest_faces(const int* __restrict__ F, long n3, const int* __restrict__ remap, int* __restrict__ dF,
                               unsigned long long* __restrict__ keys, int* __restrict__ count) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n3) return;
  const int v = remap[F[k]];
  dF[k] = v;
  keys[k] = ((unsigned long long)(unsigned)v << 32) | (unsigned long long)(k / 3);
  atomicAdd(count + v, 1);
}

__global__ void k_iota(int* __restrict__ out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = i;
}

__global__ void k_keys_low32(const unsigned long long* __restrict__ keys, long n, int* __restrict__ out) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) out[k] = (int)(unsigned)(keys[k] & 0xffffffffull);
}

// ---------------------------------------------------------------------------
// BVH, level by level
// ---------------------------------------------------------------------------
// Per triangle: bmin(3) bmax(3) centroid(3), the host builder's expressions.
__global__ void k_tri_info(const float* __restrict__ V, const int* __restrict__ F, int nF, float* __restrict__ info) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nF) return;
  const float* a = V + 3 * (size_t)F[3 * t];
  const float* b = V + 3 * (size_t)F[3 * t + 1];
  const float* c = V + 3 * (size_t)F[3 * t + 2];
  float* o = info + 9 * (size_t)t;
  const float third = 1.0f / 3.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    o[k] = fminf(a[k], fminf(b[k], c[k]));
    o[3 + k] = fmaxf(a[k], fmaxf(b[k], c[k]));
    o[6 + k] = (a[k] + (b[k] + c[k])) * third;
  }
}

// One segment of a level of the id array: its node, and the nodes of its halves.
struct BvhSeg {
  int start, count, node, left, right;
};

__device__ __forceinline__ int seg_of(const BvhSeg* __restrict__ segs, int nseg, int p) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (segs[mid].start <= p) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// acc per segment: bmin3 bmax3 cmin3 cmax3 as ord ints
__global__ void k_seg_acc_init(int nseg, int* acc) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
#pragma unroll
  for (int k = 0; k < 12; ++k) acc[12 * s + k] = (k % 6) < 3 ? INT_MAX : INT_MIN;
}

// Triangle t's box and centroid into word k of its segment's accumulators:
// lanes of one segment are reduced first (peers, of which `leader` adds).
__device__ __forceinline__ void seg_accumulate(const float* __restrict__ o, bool in, unsigned peers, bool leader, int* acc) {
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    // bmin <- tri bmin, bmax <- tri bmax, cmin/cmax <- centroid
    const int src = k < 9 ? k : k - 3;
    const bool is_min = (k % 6) < 3;
    int v = is_min ? INT_MAX : INT_MIN;
    if (in) v = ing_f2ord(o[src]);
    v = is_min ? __reduce_min_sync(peers, v) : __reduce_max_sync(peers, v);
    if (in && leader) {
      if (is_min) atomicMin(acc + k, v); else atomicMax(acc + k, v);
    }
  }
}

// A block's positions lie in one or two segments of the upper levels: summed
// in shared memory for the first two, directly for others (per-warp atomics
// on the root's twelve words took 24 us per level at 200k triangles).
__global__ void __launch_bounds__(256) k_seg_reduce(const int* __restrict__ tids, int n, const BvhSeg* __restrict__ segs,
                                                    int nseg, const float* __restrict__ info, int* __restrict__ acc) {
  __shared__ int sacc[24];
  __shared__ int s0;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (threadIdx.x < 24) sacc[threadIdx.x] = (threadIdx.x % 6) < 3 ? INT_MAX : INT_MIN;
  int s = -1;
  if (p < n) {
    s = seg_of(segs, nseg, p);
    if (threadIdx.x == 0) s0 = s;
  }
  __syncthreads();
  const unsigned peers = __match_any_sync(0xffffffffu, s);
  const bool leader = (int)(threadIdx.x & 31) == __ffs(peers) - 1;
  const int rel = s - s0;
  int* dst = s < 0 ? sacc : rel < 2 ? sacc + 12 * rel : acc + 12 * (size_t)s;
  seg_accumulate(info + 9 * (size_t)(s >= 0 ? tids[p] : 0), s >= 0, peers, leader, dst);
  __syncthreads();
  if (threadIdx.x < 24) {
    const int k = threadIdx.x % 12, v = sacc[threadIdx.x];
    const bool is_min = (k % 6) < 3;
    if (v != (is_min ? INT_MAX : INT_MIN)) {
      int* w = acc + 12 * (size_t)(s0 + threadIdx.x / 12) + k;
      if (is_min) atomicMin(w, v); else atomicMax(w, v);
    }
  }
}

// Node of segment g from its accumulators, and its split axis (-1: a leaf).
__device__ __forceinline__ int seg_node(const BvhSeg& g, const int* acc, int leaf, BVHNode* __restrict__ nodes) {
  BVHNode nd;
  int axis = -1;
#pragma unroll
  for (int a = 0; a < 3; ++a) { nd.bmin[a] = ing_ord2f(acc[a]); nd.bmax[a] = ing_ord2f(acc[3 + a]); }
  if (g.count <= leaf) {
    nd.left = nd.right = -1;
    nd.triStart = g.start;
    nd.triCount = g.count;
  } else {
    const float ex = ing_ord2f(acc[9]) - ing_ord2f(acc[6]);
    const float ey = ing_ord2f(acc[10]) - ing_ord2f(acc[7]);
    const float ez = ing_ord2f(acc[11]) - ing_ord2f(acc[8]);
    axis = (ex >= ey && ex >= ez) ? 0 : (ey >= ez ? 1 : 2);
    nd.left = g.left;
    nd.right = g.right;
    nd.triStart = -1;
    nd.triCount = 0;
  }
  nodes[g.node] = nd;
  return axis;
}

// centroid coordinate as a sort key (-0 folded into +0, monotone unsigned map)
__device__ __forceinline__ unsigned centroid_key(const float* __restrict__ info, int tri, int axis) {
  const unsigned u = __float_as_uint(info[9 * (size_t)tri + 6 + axis] + 0.0f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Nodes of an upper level (pre-order slots), whose segments all split, and the
// split axis of each.
__global__ void k_seg_emit(const BvhSeg* __restrict__ segs, int nseg, const int* __restrict__ acc, int leaf,
                           BVHNode* __restrict__ nodes, int* __restrict__ axis) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  axis[s] = seg_node(segs[s], acc + 12 * (size_t)s, leaf, nodes);
}

// sort keys: segment rank in the high word, then the centroid coordinate on the
// segment's axis (-0 folded into +0, monotone unsigned map)
__global__ void k_seg_keys(const int* __restrict__ tids, int n, const BvhSeg* __restrict__ segs, int nseg,
                           const int* __restrict__ axis, const float* __restrict__ info,
                           unsigned long long* __restrict__ keys) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int s = seg_of(segs, nseg, p);
  keys[p] = ((unsigned long long)(unsigned)s << 32) | centroid_key(info, tids[p], axis[s]);
}

// ---------------------------------------------------------------------------
// The lower levels: one block finishes the subtree of a segment of at most
// kSubTris triangles in shared memory, level by level like the steps above.
// The order within a segment comes from a bitonic sort of (segment,
// coordinate, position) keys; the position makes every key distinct and the
// order that of a stable sort.  Bound by barriers and shuffles; 128 subtrees of
// 1562 triangles: 165 us (225 with every step of the sort through shared
// memory); the same nine levels over all triangles took 1.3 ms in launches.
// ---------------------------------------------------------------------------
constexpr int kSubTris = 2048;
constexpr int kSubThreads = 1024;
constexpr int kSubSegs = kSubTris / 4 + 1;  // a split segment's halves hold at least 4

struct SubTree {
  unsigned long long key[kSubTris];
  int tid[2][kSubTris];
  uint16_t seg[2][kSubTris];
  int acc[kSubSegs][12];
  int start[2][kSubSegs], count[2][kSubSegs], node[2][kSubSegs];
  int axis[kSubSegs], next[kSubSegs];
  int warp[33];
  int nseg;
};

// subtree: nodes of the subtree of n triangles, for n <= kSubTris
__global__ void __launch_bounds__(kSubThreads) k_bvh_subtree(int* __restrict__ tids, const BvhSeg* __restrict__ segs,
                                                             const float* __restrict__ info, const int* __restrict__ subtree,
                                                             int leaf, BVHNode* __restrict__ nodes) {
  extern __shared__ __align__(16) unsigned char sub_raw[];
  SubTree& T = *reinterpret_cast<SubTree*>(sub_raw);
  const BvhSeg top = segs[blockIdx.x];
  const int n = top.count, tx = threadIdx.x;
  int pad = 64;  // elements sorted (a power of two; thread t holds 2t and 2t + 1)
  while (pad < n) pad <<= 1;
  for (int p = tx; p < n; p += kSubThreads) { T.tid[0][p] = tids[top.start + p]; T.seg[0][p] = 0; }
  if (tx == 0) { T.start[0][0] = 0; T.count[0][0] = n; T.node[0][0] = top.node; T.nseg = 1; }
  __syncthreads();
  for (int cur = 0;; cur ^= 1) {
    const int nseg = T.nseg;
    for (int k = tx; k < 12 * nseg; k += kSubThreads) T.acc[k / 12][k % 12] = (k % 6) < 3 ? INT_MAX : INT_MIN;
    __syncthreads();
    for (int p0 = 0; p0 < n; p0 += kSubThreads) {
      const int p = p0 + tx;
      int s = -1;
      if (p < n) {
        s = T.seg[cur][p];
        if (T.node[cur][s] < 0) s = -1;
      }
      const unsigned peers = __match_any_sync(0xffffffffu, s);
      seg_accumulate(info + 9 * (size_t)(s >= 0 ? T.tid[cur][p] : 0), s >= 0, peers, (tx & 31) == __ffs(peers) - 1,
                     T.acc[s >= 0 ? s : 0]);
    }
    __syncthreads();
    // nodes; places of the next level's segments (a split one becomes two)
    int mine = 0;
    if (tx < nseg) {
      T.axis[tx] = -1;
      const int nd = T.node[cur][tx], c = T.count[cur][tx];
      if (nd >= 0) {
        const BvhSeg g{top.start + T.start[cur][tx], c, nd, nd + 1, c > leaf ? nd + 1 + subtree[c / 2] : -1};
        T.axis[tx] = seg_node(g, T.acc[tx], leaf, nodes);
      }
      mine = T.axis[tx] >= 0 ? 2 : 1;
    }
    int total;
    const int at = block_exclusive_scan(mine, T.warp, total);
    if (total == nseg) {  // no segment splits
      for (int p = tx; p < n; p += kSubThreads) tids[top.start + p] = T.tid[cur][p];
      return;
    }
    if (tx < nseg) {
      const int st = T.start[cur][tx], c = T.count[cur][tx], nd = T.node[cur][tx];
      T.next[tx] = at;
      if (mine == 2) {
        T.start[cur ^ 1][at] = st; T.count[cur ^ 1][at] = c / 2; T.node[cur ^ 1][at] = nd + 1;
        T.start[cur ^ 1][at + 1] = st + c / 2; T.count[cur ^ 1][at + 1] = c - c / 2;
        T.node[cur ^ 1][at + 1] = nd + 1 + subtree[c / 2];
      } else {
        T.start[cur ^ 1][at] = st; T.count[cur ^ 1][at] = c; T.node[cur ^ 1][at] = -1;
      }
    }
    if (tx == 0) T.nseg = total;
    // thread t sorts elements 2t and 2t + 1: exchanges within a warp's 64
    // elements by shuffles, wider ones through shared memory
    unsigned long long e[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int p = 2 * tx + r;
      e[r] = ~0ull;
      if (p < n) {
        const int s = T.seg[cur][p], ax = T.axis[s];
        const unsigned lo = ax >= 0 ? centroid_key(info, T.tid[cur][p], ax) : 0u;
        e[r] = ((unsigned long long)s << 43) | ((unsigned long long)lo << 11) | (unsigned long long)p;
      }
    }
    for (int kk = 2; kk <= pad; kk <<= 1) {
      const bool up = ((2 * tx) & kk) == 0;
      for (int j = kk >> 1; j >= 64; j >>= 1) {
        __syncthreads();
        T.key[2 * tx] = e[0]; T.key[2 * tx + 1] = e[1];
        __syncthreads();
        const bool low = ((2 * tx) & j) == 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const unsigned long long o = T.key[(2 * tx + r) ^ j];
          e[r] = (low == up) == (e[r] < o) ? e[r] : o;
        }
      }
      for (int j = min(kk >> 1, 32); j >= 2; j >>= 1) {
        const bool low = ((2 * tx) & j) == 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const unsigned long long o = __shfl_xor_sync(0xffffffffu, e[r], j >> 1);
          e[r] = (low == up) == (e[r] < o) ? e[r] : o;
        }
      }
      // the pair itself (for kk == 2 the direction alternates with the pair)
      const bool pup = kk == 2 ? (tx & 1) == 0 : up;
      if ((e[0] > e[1]) == pup) { const unsigned long long x = e[0]; e[0] = e[1]; e[1] = x; }
    }
    __syncthreads();
    T.key[2 * tx] = e[0]; T.key[2 * tx + 1] = e[1];
    __syncthreads();
    for (int q = tx; q < n; q += kSubThreads) {
      const unsigned long long k = T.key[q];
      const int p = (int)(k & 2047u), s = (int)(k >> 43);
      T.tid[cur ^ 1][q] = T.tid[cur][p];
      T.seg[cur ^ 1][q] = (uint16_t)(T.next[s] + (T.axis[s] >= 0 && q - T.start[cur][s] >= T.count[cur][s] / 2 ? 1 : 0));
    }
    __syncthreads();
  }
}

// The tree as the traversals read it (BvhView), one node per thread.
__global__ void k_bvh_pack(const BVHNode* __restrict__ nodes, int n_nodes, const int* __restrict__ tids,
                           const float* __restrict__ V, const int* __restrict__ F, float4* __restrict__ pair,
                           float4* __restrict__ tris) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_nodes) return;
  const BVHNode nd = nodes[i];
  if (nd.triCount > 0) {
    for (int k = 0; k < nd.triCount; ++k) {
      const long t = (long)nd.triStart + k;
      const int f = tids[t];
      const V3<float> a = ld3(V, F[3 * (long)f]), b = ld3(V, F[3 * (long)f + 1]), c = ld3(V, F[3 * (long)f + 2]);
      tris[3 * t] = make_float4(a.x, a.y, a.z, b.x);
      tris[3 * t + 1] = make_float4(b.y, b.z, c.x, c.y);
      tris[3 * t + 2] = make_float4(c.z, __int_as_float(k + 1 == nd.triCount ? 1 : 0), 0.f, 0.f);
    }
    return;
  }
  const BVHNode l = nodes[nd.left], r = nodes[nd.right];
  float4* w = pair + 4 * (size_t)i;
  w[0] = make_float4(l.bmin[0], l.bmin[1], l.bmin[2], l.bmax[0]);
  w[1] = make_float4(l.bmax[1], l.bmax[2], r.bmin[0], r.bmin[1]);
  w[2] = make_float4(r.bmin[2], r.bmax[0], r.bmax[1], r.bmax[2]);
  w[3] = make_float4(__int_as_float(l.triCount > 0 ? ~l.triStart : nd.left),
                     __int_as_float(r.triCount > 0 ? ~r.triStart : nd.right), 0.f, 0.f);
}

}  // namespace cvt
