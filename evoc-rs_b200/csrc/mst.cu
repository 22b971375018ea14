// Borůvka minimum spanning tree under mutual-reachability distance, with the
// core distances, on the GPU.
//
// Replaces build_kdtree (src/kdtree.rs:367-413), parallel_tree_query
// (src/kdtree.rs:592-629), initialize_boruvka_from_knn and parallel_boruvka
// with reproducible = false (src/boruvka.rs:437-593): the MST that
// build_cluster_layers (src/clustering.rs:50-110) condenses into the cluster
// hierarchy, over the node embedding (n points of 4..15 dimensions there).
//
//   rdist(a, b)   squared Euclidean distance, summed serially over the
//                 dimensions in f32 without contraction (src/kdtree.rs:415-423)
//   core[i]       rdist to the (min_samples + 1)-th nearest point, the point
//                 itself included (parallel_tree_query with output_rdist)
//   mr(i, j)      max(rdist(i, j), core[i], core[j])
//   edges         n - 1 rows (from, to, sqrt(mr)) as f32, in the order found
//
// Tree.  The reference's balanced KD-tree: node i has children 2i+1 and 2i+2,
// n_levels = floor(log2(max(n-1, 1) / leaf_size)) + 1, and every node's
// positions are fixed by halving -- [s, e) splits at s + (e-s)/2 -- so only
// which points fill a range depends on the data.  It is built level by level:
// each node's bounds (block per node), its split dimension (largest spread,
// first on ties, src/kdtree.rs:232-257), then one stable radix sort of
// (node, coordinate on the node's split dimension) keys puts every node's
// lower half left of its median, as the reference's introselect does (the
// order inside the halves may differ; the tree's geometry does not).  Subtrees
// that fit shared memory are finished by one block each, and the leaves are
// smaller than the reference's 40 to 79 points: the results do not depend on
// where the tree stops.  Points
// are then stored in tree order, so a leaf is a contiguous run.
//
// Queries.  A warp walks the tree for 32 points that follow each other in tree
// order (or, in a Borůvka round with few points left, for one), visits the
// nearer child first, as the reference's recursion does, and prunes on the node
// lower bound (point_to_node_lower_bound_rdist, src/kdtree.rs:425-447).
//
// Borůvka.  Components live in a lock-free union-find over tree positions.
// The kNN initialisation takes, for each point, the first of its sorted
// neighbours j >= 1 with core[i] >= core[j] (src/boruvka.rs:437-477).  Each
// round every point that can still lower its component's bound (see Known)
// searches for its nearest point in another component under mr, pruning nodes whose points all share its component (node components,
// src/boruvka.rs:88-127), nodes farther than its best so far, and nodes
// farther than its component's shared bound (an atomic minimum, as the
// non-reproducible reference keeps it, src/boruvka.rs:262-318).  Each
// component's candidate is the smallest (mr, point) key of its points -- the
// lowest point among equal distances, as merge_components keeps the first --
// and components are joined by CAS union; an edge is kept only when its union
// links two roots.  A cycle among the components' choices can only join
// edges of one equal weight, so dropping the closing edge keeps an MST: the
// result has the reference's total weight and the same sorted weights; edges
// can differ only among equal weights.  The reproducible mode
// (boruvka_tree_query_reproducible) freezes component bounds block by block in
// point order and is serial at the block level; it is not built here.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/evoc_gpu.h"
#include "common.cuh"
#include "ctx.h"

namespace evoc {
namespace mst {

constexpr int kMaxStack = 64;  // > 2 * levels: a visit pushes two children and pops one
constexpr int kMaxKnn = 32;    // min_samples + 1
constexpr int kLeafSize = 16;  // to 31 points: a step of a warp
constexpr uint32_t kInfBits = 0x7f800000u;

struct TreeView {
  int64_t n;
  int n_nodes;
  const int32_t* order;  // tree position -> point index
  const float* pts;      // points in tree order, P floats each (zero padded)
  const int32_t* nstart;
  const int32_t* nend;
  int first_leaf;        // nodes from here on are the leaves, the tree's last level
  const float* lo;       // per node, P floats
  const float* hi;
};

template <int P>
__device__ __forceinline__ void load_point(const float* __restrict__ src, float (&q)[P]) {
  const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll
  for (int c = 0; c < P / 4; c++) {
    const float4 v = s4[c];
    q[4 * c] = v.x;
    q[4 * c + 1] = v.y;
    q[4 * c + 2] = v.z;
    q[4 * c + 3] = v.w;
  }
}

// rdist in the reference's order; zero-padded dimensions add +0.0 exactly.
template <int P>
__device__ __forceinline__ float rdist(const float (&q)[P], const float* __restrict__ y) {
  float y4[P];
  load_point<P>(y, y4);
  float r = 0.0f;
#pragma unroll
  for (int c = 0; c < P; c++) {
    const float d = __fsub_rn(q[c], y4[c]);
    r = __fadd_rn(r, __fmul_rn(d, d));
  }
  return r;
}

template <int P>
__device__ __forceinline__ float node_lower_bound(const float (&q)[P], const float* __restrict__ lo,
                                                  const float* __restrict__ hi) {
  float r = 0.0f;
#pragma unroll
  for (int c = 0; c < P; c++) {
    const float dl = lo[c] > q[c] ? __fsub_rn(lo[c], q[c]) : 0.0f;
    const float dh = q[c] > hi[c] ? __fsub_rn(q[c], hi[c]) : 0.0f;
    const float d = __fadd_rn(dl, dh);
    r = __fadd_rn(r, __fmul_rn(d, d));
  }
  return r;
}

// ------------------------------------------------------------------ tree build

__global__ void pad_points_kernel(const float* __restrict__ X, int64_t n, int dim, int64_t ldx, float* __restrict__ Xp,
                                  int P) {
  const int64_t total = n * P;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e / P;
    const int c = int(e % P);
    Xp[e] = c < dim ? X[i * ldx + c] : 0.0f;
  }
}

__global__ void iota_kernel(int32_t* __restrict__ a, int64_t n) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    a[i] = int32_t(i);
}

// Minima and maxima over the lanes of a warp.
template <int P>
__device__ __forceinline__ void warp_bounds(float (&mn)[P], float (&mx)[P]) {
#pragma unroll
  for (int c = 0; c < P; c++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn[c] = fminf(mn[c], __shfl_xor_sync(0xffffffffu, mn[c], o));
      mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
    }
  }
}

// Bounds of the `count` nodes from `first` on, each read by gridDim.x blocks:
// a level near the root has fewer nodes than the chip has SMs, and its one
// block a node took most of the build.  The blocks meet in atomics on words
// that order as their floats do.
template <int P>
__global__ void __launch_bounds__(256) node_bounds_kernel(const float* __restrict__ Xp,
                                                          const int32_t* __restrict__ order,
                                                          const int32_t* __restrict__ nstart,
                                                          const int32_t* __restrict__ nend, int first, int count,
                                                          uint32_t* __restrict__ lo, uint32_t* __restrict__ hi) {
  for (int b = blockIdx.y; b < count; b += gridDim.y) {
    const int node = first + b;
    const int32_t s = nstart[node], e = nend[node];
    float mn[P], mx[P];
#pragma unroll
    for (int c = 0; c < P; c++) {
      mn[c] = __int_as_float(0x7f800000);
      mx[c] = __int_as_float(0xff800000);
    }
    for (int64_t p = int64_t(s) + blockIdx.x * 256 + threadIdx.x; p < e; p += int64_t(gridDim.x) * 256) {
      float v[P];
      load_point<P>(Xp + int64_t(order[p]) * P, v);
#pragma unroll
      for (int c = 0; c < P; c++) {
        mn[c] = fminf(mn[c], v[c]);
        mx[c] = fmaxf(mx[c], v[c]);
      }
    }
    warp_bounds<P>(mn, mx);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int c = 0; c < P; c++) {
        atomicMin(&lo[int64_t(node) * P + c], orderable(mn[c]));
        atomicMax(&hi[int64_t(node) * P + c], orderable(mx[c]));
      }
  }
}

// A level's bounds as floats, and its split dimensions.
template <int P>
__global__ void node_split_kernel(int first, int count, int dim, uint32_t* __restrict__ lo, uint32_t* __restrict__ hi,
                                  int32_t* __restrict__ split) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < count; b += gridDim.x * blockDim.x) {
    const int64_t at = int64_t(first + b) * P;
    float l[P], h[P];
#pragma unroll
    for (int c = 0; c < P; c++) {
      l[c] = from_orderable(lo[at + c]);
      h[c] = from_orderable(hi[at + c]);
      lo[at + c] = __float_as_uint(l[c]);
      hi[at + c] = __float_as_uint(h[c]);
    }
    int best = 0;
    float spread_max = 0.0f;
#pragma unroll
    for (int c = 0; c < P; c++) {
      const float spread = __fsub_rn(h[c], l[c]);
      if (c < dim && spread > spread_max) {
        spread_max = spread;
        best = c;
      }
    }
    split[first + b] = best;
  }
}

// Sort keys of one level: (node within the level, coordinate on its split dimension).
__global__ void split_keys_kernel(const float* __restrict__ Xp, int P, const int32_t* __restrict__ order, int64_t n,
                                  const int32_t* __restrict__ nstart, int first, int count,
                                  const int32_t* __restrict__ split, uint64_t* __restrict__ keys) {
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {  // last node of the level starting at or before p
      const int mid = (lo + hi + 1) >> 1;
      if (nstart[first + mid] <= p) lo = mid;
      else hi = mid - 1;
    }
    const float v = Xp[int64_t(order[p]) * P + split[first + lo]];
    keys[p] = (uint64_t(uint32_t(lo)) << 32) | uint64_t(orderable(v));
  }
}

// The rest of the tree below one node of level `level`, whose points fit
// shared memory: bounds, split dimensions and sorts of all its levels in one
// block, then its points in tree order.  A sort's keys are (node, coordinate,
// point), so equal coordinates keep an order of their own.
// 300,000 x 7 (256 subtrees of 1,172 points): 0.38 ms for seven levels, where
// a level took a launch for the bounds and a radix sort of all points, 0.15 ms.
template <int P>
struct Subtree {
  static constexpr int kCap = P <= 16 ? 2048 : 1024;
  static constexpr int kThreads = P <= 8 ? 1024 : 512;
  static constexpr size_t kSmem = size_t(kCap) * (P * 4 + 8 + 4 + 2);
};

template <int P>
__global__ void __launch_bounds__(Subtree<P>::kThreads) subtree_kernel(const float* __restrict__ Xp, int32_t* __restrict__ order,
                                                       const int32_t* __restrict__ nstart,
                                                       const int32_t* __restrict__ nend, int level, int n_levels,
                                                       int dim, float* __restrict__ lo, float* __restrict__ hi,
                                                       float* __restrict__ pts) {
  constexpr int kCap = Subtree<P>::kCap;
  extern __shared__ __align__(16) unsigned char smem[];
  float* X = reinterpret_cast<float*>(smem);
  uint64_t* key = reinterpret_cast<uint64_t*>(smem + size_t(kCap) * P * 4);
  int32_t* ids = reinterpret_cast<int32_t*>(key + kCap);
  uint16_t* perm = reinterpret_cast<uint16_t*>(ids + kCap);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  const int root = (1 << level) - 1 + blockIdx.x;
  const int32_t s0 = nstart[root];
  const int m = nend[root] - s0;
  int width = 2;  // of the sort
  while (width < m) width <<= 1;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const int32_t id = order[s0 + i];
    ids[i] = id;
    perm[i] = uint16_t(i);
    const float4* src = reinterpret_cast<const float4*>(Xp + int64_t(id) * P);
#pragma unroll
    for (int c = 0; c < P / 4; c++) reinterpret_cast<float4*>(X)[i * (P / 4) + c] = src[c];
  }
  __syncthreads();
  for (int l = level; l < n_levels; l++) {
    const bool last = l == n_levels - 1;
    const int first = ((root + 1) << (l - level)) - 1;
    for (int j = warp; j < (1 << (l - level)); j += n_warps) {
      const int node = first + j;
      const int a = nstart[node] - s0, e = nend[node] - s0;
      float mn[P], mx[P];
#pragma unroll
      for (int c = 0; c < P; c++) {
        mn[c] = __int_as_float(0x7f800000);
        mx[c] = __int_as_float(0xff800000);
      }
      for (int i = a + lane; i < e; i += 32) {
        float v[P];
        load_point<P>(X + int(perm[i]) * P, v);
#pragma unroll
        for (int c = 0; c < P; c++) {
          mn[c] = fminf(mn[c], v[c]);
          mx[c] = fmaxf(mx[c], v[c]);
        }
      }
      warp_bounds<P>(mn, mx);
      int split = 0;
      float spread_max = 0.0f;
#pragma unroll
      for (int c = 0; c < P; c++) {
        const float spread = __fsub_rn(mx[c], mn[c]);
        if (c < dim && spread > spread_max) {
          spread_max = spread;
          split = c;
        }
        if (lane == 0) {
          lo[int64_t(node) * P + c] = mn[c];
          hi[int64_t(node) * P + c] = mx[c];
        }
      }
      if (!last)
        for (int i = a + lane; i < e; i += 32)
          key[i] = (uint64_t(j) << 43) | (uint64_t(orderable(X[int(perm[i]) * P + split])) << 11) | perm[i];
    }
    if (last) break;
    for (int i = m + threadIdx.x; i < width; i += blockDim.x) key[i] = ~0ull;
    __syncthreads();
    for (int len = 2; len <= width; len <<= 1)
      for (int half = len >> 1; half > 0; half >>= 1) {
        for (int t = threadIdx.x; t < width / 2; t += blockDim.x) {
          const int i = 2 * half * (t / half) + t % half;
          const uint64_t x = key[i], y = key[i + half];
          if ((x > y) == ((i & len) == 0)) {
            key[i] = y;
            key[i + half] = x;
          }
        }
        __syncthreads();
      }
    for (int i = threadIdx.x; i < m; i += blockDim.x) perm[i] = uint16_t(key[i] & 2047);
    __syncthreads();
  }
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const int at = perm[i];
    order[s0 + i] = ids[at];
    float4* dst = reinterpret_cast<float4*>(pts + int64_t(s0 + i) * P);
#pragma unroll
    for (int c = 0; c < P / 4; c++) dst[c] = reinterpret_cast<const float4*>(X)[at * (P / 4) + c];
  }
}

// ------------------------------------------------------------------ walks

// A walk is a warp's: its 32 lanes hold 32 points that lie close together, the
// warp visits a node when any lane can find something in it, and every lane
// tests every point of a visited leaf.  Nodes, boxes and points are the same
// address for the whole warp, so a visit costs one transaction where a stack
// per thread cost 32, and no lane waits for another's branch.  The price is
// the union of the lanes' paths; leaves of 16 to 31 points keep it small.
//
// `best()` of a lane is the distance above which it has no use for a node
// (-infinity: the lane is finished), `floor` a lower bound of every distance
// it can find.  `leaf(node, want)` tests a leaf's points.
template <int P, class Best, class Skip, class Leaf>
__device__ __forceinline__ void warp_walk(const TreeView& t, const float (&q)[P], float floor_d, Best best, Skip skip,
                                          Leaf leaf, int* __restrict__ status) {
  int sn[kMaxStack];
  float sl[kMaxStack];
  int sp = 0;
  sn[0] = 0;
  sl[0] = fmaxf(floor_d, node_lower_bound<P>(q, t.lo, t.hi));
  sp = 1;
  while (sp > 0) {
    const int node = sn[--sp];
    const float lb = sl[sp];
    const float thr = best();
    // while nothing is known every node is open, boxes at infinity too
    const bool want = (lb < thr || thr == __int_as_float(0x7f800000)) && !skip(node);
    const unsigned wants = __ballot_sync(0xffffffffu, want);
    if (wants == 0u) continue;
    if (node >= t.first_leaf) {
      leaf(node, want);
      continue;
    }
    const int l = 2 * node + 1, r = l + 1;
    const float bl = fmaxf(floor_d, node_lower_bound<P>(q, t.lo + int64_t(l) * P, t.hi + int64_t(l) * P));
    const float br = fmaxf(floor_d, node_lower_bound<P>(q, t.lo + int64_t(r) * P, t.hi + int64_t(r) * P));
    if (sp + 2 > kMaxStack) {  // cannot happen for the checked depths; stop rather than overrun
      atomicCAS(status, 0, 1);
      break;
    }
    // the child that more of the interested lanes are nearer to is visited first (pushed last)
    const bool left = 2 * __popc(__ballot_sync(0xffffffffu, want && bl <= br)) >= __popc(wants);
    sn[sp] = left ? r : l;
    sl[sp++] = left ? br : bl;
    sn[sp] = left ? l : r;
    sl[sp++] = left ? bl : br;
  }
}

// ------------------------------------------------------------------ k-NN query (core distances)

// Lane per tree position: the kq nearest positions (self included), sorted by
// (rdist, position); core = the kq-th rdist.  The neighbours are KQ sorted
// registers, the first KQ - kq of them below every distance, so the last one
// is the kq-th nearest whatever kq is.
//
// Bound by instructions: a warp tests a point in 3 P of them, and the union of
// its lanes' paths is most of their cluster.  300,000 x 7, kq 6: 7.9 ms with a
// stack and a binary heap per thread, 5.0 ms now, 69 % of the issue slots used.
template <int P, int KQ>
__global__ void __launch_bounds__(128) knn_kernel(TreeView t, int kq, float* __restrict__ core,
                                                  int32_t* __restrict__ knn_pos, float* __restrict__ knn_d,
                                                  int* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const int64_t n_warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t w = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); 32 * w < t.n; w += n_warps) {
    const int64_t p = 32 * w + lane;
    const bool live = p < t.n;
    float q[P];
    load_point<P>(t.pts + (live ? p : t.n - 1) * P, q);
    float hd[KQ];
    int32_t hp[KQ];
#pragma unroll
    for (int j = 0; j < KQ; j++) {
      hd[j] = live && j >= KQ - kq ? __int_as_float(0x7f800000) : __int_as_float(0xff800000);
      hp[j] = -1;
    }
    warp_walk<P>(
        t, q, 0.0f, [&] { return hd[KQ - 1]; }, [](int) { return false; },
        [&](int node, bool) {
          const int32_t e = t.nend[node];
#pragma unroll 4
          for (int32_t s = t.nstart[node]; s < e; s++) {
            const float d = rdist<P>(q, t.pts + int64_t(s) * P);
            if (d < hd[KQ - 1]) {
#pragma unroll
              for (int j = KQ - 1; j > 0; j--) {
                const bool up = d < hd[j - 1];
                const bool here = d < hd[j];
                hp[j] = up ? hp[j - 1] : here ? s : hp[j];
                hd[j] = up ? hd[j - 1] : here ? d : hd[j];
              }
              if (d < hd[0]) {
                hd[0] = d;
                hp[0] = s;
              }
            }
          }
        },
        status);
    if (!live) continue;
    core[p] = hd[KQ - 1];
    // equal distances by position (they stand in the order of the visits)
    bool swapped = true;
    while (swapped) {
      swapped = false;
#pragma unroll
      for (int j = 1; j < KQ; j++) {
        if (j > KQ - kq && hd[j] == hd[j - 1] && uint32_t(hp[j]) < uint32_t(hp[j - 1])) {
          const int32_t x = hp[j];
          hp[j] = hp[j - 1];
          hp[j - 1] = x;
          swapped = true;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < KQ; j++) {
      if (j >= KQ - kq) {
        knn_pos[p * kq + j - (KQ - kq)] = hp[j];
        knn_d[p * kq + j - (KQ - kq)] = hd[j];
      }
    }
  }
}

// ------------------------------------------------------------------ union-find over tree positions

__device__ __forceinline__ int32_t uf_find(int32_t* parent, int32_t x) {
  for (;;) {
    const int32_t p = reinterpret_cast<volatile int32_t*>(parent)[x];
    const int32_t g = reinterpret_cast<volatile int32_t*>(parent)[p];
    if (p == g) return p;
    atomicCAS(&parent[x], p, g);  // path halving
    x = g;
  }
}

// Links the roots of a and b (larger under smaller); false when already joined.
__device__ __forceinline__ bool uf_unite(int32_t* parent, int32_t a, int32_t b) {
  for (;;) {
    a = uf_find(parent, a);
    b = uf_find(parent, b);
    if (a == b) return false;
    if (a < b) {
      const int32_t t = a;
      a = b;
      b = t;
    }
    if (atomicCAS(&parent[a], a, b) == a) return true;
  }
}

__device__ __forceinline__ void add_edge(int32_t a, int32_t b, float w, int32_t* __restrict__ e_from,
                                         int32_t* __restrict__ e_to, float* __restrict__ e_w, int32_t* count,
                                         int64_t cap) {
  const int32_t slot = atomicAdd(count, 1);
  if (slot < cap) {
    e_from[slot] = a;
    e_to[slot] = b;
    e_w[slot] = w;
  }
}

// initialize_boruvka_from_knn (src/boruvka.rs:437-477): each point's first
// sorted neighbour j >= 1 with core[i] >= core[j], joined when it links two
// components.  (The reference joins them serially in point order; any
// spanning forest of these edges has the same weight: each is a minimum
// mutual-reachability edge of its point, and a cycle among them has equal
// weights.)
__global__ void knn_init_kernel(int64_t n, int kq, const float* __restrict__ core, const int32_t* __restrict__ knn_pos,
                                const float* __restrict__ knn_d, int32_t* __restrict__ parent,
                                int32_t* __restrict__ e_from, int32_t* __restrict__ e_to, float* __restrict__ e_w,
                                int32_t* count, int64_t cap) {
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    for (int j = 1; j < kq; j++) {
      const int32_t nb = knn_pos[p * kq + j];
      if (nb < 0) break;
      if (core[p] >= core[nb]) {
        const float w = fmaxf(core[p], knn_d[p * kq + j]);
        if (uf_unite(parent, int32_t(p), nb)) add_edge(int32_t(p), nb, w, e_from, e_to, e_w, count, cap);
        break;
      }
    }
  }
}

// What a point knows from one round to the next.  Components only grow, so
// `low` (no point outside its component is nearer, under mutual reachability)
// stays true, and the nearest one found so far (`near_pos`, `near_d`) is a
// candidate for as long as it lies in another component.
struct Known {
  float* low;
  int32_t* near_pos;
  float* near_d;
};

__global__ void known_init_kernel(int64_t n, const float* __restrict__ core, Known k) {
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    k.low[p] = core[p];
    k.near_pos[p] = -1;
    k.near_d[p] = __int_as_float(0x7f800000);
  }
}

// A round's components, with their bounds and candidates cleared.
__global__ void components_kernel(int64_t n, int32_t* __restrict__ parent, int32_t* __restrict__ comp,
                                  uint32_t* __restrict__ bound, unsigned long long* __restrict__ best) {
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    const int32_t r = uf_find(parent, int32_t(p));
    comp[p] = r;
    parent[p] = r;
    bound[p] = kInfBits;
    best[p] = ~0ull;
  }
}

// Node components (src/boruvka.rs:101-126): a leaf whose points share one
// component has it, an internal node whose children have the same value has
// it, else -1; and once, with `core`, the smallest core distance below each
// node.  Thread per leaf; the second of two children to arrive goes on to
// their parent (`arrived` gains two a call, so it needs no clearing).
__global__ void node_values_kernel(TreeView t, const int32_t* __restrict__ comp, int32_t* node_comp,
                                   const float* __restrict__ core, float* node_core, int32_t* __restrict__ arrived) {
  const int node0 = t.first_leaf + blockIdx.x * blockDim.x + threadIdx.x;
  if (node0 >= t.n_nodes) return;
  const int32_t s = t.nstart[node0], e = t.nend[node0];
  if (core) {
    float m = __int_as_float(0x7f800000);
    for (int32_t p = s; p < e; p++) m = fminf(m, core[p]);
    node_core[node0] = m;
  } else {
    int32_t c = s < e ? comp[s] : -1;
    for (int32_t p = s + 1; p < e; p++)
      if (comp[p] != c) c = -1;
    node_comp[node0] = c;
  }
  for (int node = node0; node > 0;) {
    node = (node - 1) >> 1;
    __threadfence();
    if ((atomicAdd(&arrived[node], 1) & 1) == 0) return;
    __threadfence();
    const int l = 2 * node + 1, r = l + 1;
    if (core) {
      volatile float* v = node_core;
      v[node] = fminf(v[l], v[r]);
    } else {
      volatile int32_t* v = node_comp;
      const int32_t a = v[l], b = v[r];
      v[node] = a == b ? a : -1;
    }
  }
}

// Candidates that are still in another component; where there is none, the
// nearest of the point's kNN that is.  Each lowers its component's bound.
__global__ void seed_kernel(int64_t n, int kq, const int32_t* __restrict__ comp, const float* __restrict__ core,
                            const int32_t* __restrict__ knn_pos, const float* __restrict__ knn_d, Known k,
                            uint32_t* __restrict__ bound, unsigned long long* __restrict__ best) {
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    const int32_t c = comp[p];
    int32_t j = k.near_pos[p];
    float d = k.near_d[p];
    if (j < 0 || comp[j] == c) {
      j = -1;
      d = __int_as_float(0x7f800000);
      for (int a = 1; a < kq; a++) {
        const int32_t b = knn_pos[p * kq + a];
        if (b < 0) break;
        if (comp[b] == c) continue;
        const float m = fmaxf(fmaxf(knn_d[p * kq + a], core[p]), core[b]);
        if (m < d) {
          d = m;
          j = b;
        }
      }
      k.near_pos[p] = j;
      k.near_d[p] = d;
    }
    if (j < 0) continue;
    const uint32_t bits = __float_as_uint(d);  // non-negative floats order as their bits
    const unsigned long long key = (static_cast<unsigned long long>(bits) << 32) | uint32_t(p);
    // most of a large component's points cannot lower what is there already
    if (key < reinterpret_cast<volatile unsigned long long*>(best)[c]) {
      atomicMin(&bound[c], bits);
      atomicMin(&best[c], key);
    }
  }
}

// The points that may still lower their component's bound, in runs of 256.
__global__ void __launch_bounds__(256) open_points_kernel(int64_t n, const int32_t* __restrict__ comp,
                                                          const float* __restrict__ low,
                                                          const uint32_t* __restrict__ bound,
                                                          int32_t* __restrict__ open, int32_t* __restrict__ n_open) {
  __shared__ int sums[8];
  __shared__ int base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t s = int64_t(blockIdx.x) * 256; s < n; s += int64_t(gridDim.x) * 256) {
    const int64_t p = s + threadIdx.x;
    const bool is = p < n && low[p] < __uint_as_float(bound[comp[p]]);
    const unsigned m = __ballot_sync(0xffffffffu, is);
    if (lane == 0) sums[warp] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
      int total = 0;
      for (int w = 0; w < 8; w++) {
        const int c = sums[w];
        sums[w] = total;
        total += c;
      }
      base = total ? atomicAdd(n_open, total) : 0;
    }
    __syncthreads();
    if (is) open[base + sums[warp] + __popc(m & ((1u << lane) - 1u))] = int32_t(p);
    __syncthreads();
  }
}

// One Borůvka round's search: for every open point the nearest position of
// another component under mutual reachability (component_aware_query_recursion,
// src/boruvka.rs:131-253), with the component's shared bound.  Nodes are also
// left out by the smallest core distance below them, and a point whose
// candidate is as near as its own core distance is finished.
struct Round {
  TreeView t;
  const float* core;
  const int32_t* comp;
  const int32_t* node_comp;
  const float* node_core;
  const int32_t* open;
  int32_t* next;  // the work counter
  Known k;
  uint32_t* bound;
  unsigned long long* best;
  int* status;
};

__device__ __forceinline__ float shared_bound(const Round& r, int32_t c) {
  return __uint_as_float(reinterpret_cast<volatile uint32_t*>(r.bound)[c]);
}

// What a search found (bj < 0: nothing nearer than the candidate it started
// with).  What was left out is no nearer than the smaller of the two bounds.
__device__ __forceinline__ void keep_found(const Round& r, int32_t p, int32_t c, float bd, int32_t bj, float cbound) {
  r.k.low[p] = fmaxf(r.k.low[p], fminf(bd, cbound));
  if (bj < 0) return;
  r.k.near_pos[p] = bj;
  r.k.near_d[p] = bd;
  if (bd <= cbound) {
    atomicMin(&r.bound[c], __float_as_uint(bd));
    atomicMin(&r.best[c], (static_cast<unsigned long long>(__float_as_uint(bd)) << 32) | uint32_t(p));
  }
}

// 32 open points a warp.
template <int P>
__device__ void search_many(const Round& r, int32_t count) {
  const TreeView& t = r.t;
  const int lane = threadIdx.x & 31;
  const float inf = __int_as_float(0x7f800000);
  for (;;) {
    int32_t w = 0;
    if (lane == 0) w = atomicAdd(r.next, 32);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (uint32_t(w) >= uint32_t(count)) break;
    const int32_t p = r.open[w + lane < count ? w + lane : w];
    const int32_t c = r.comp[p];
    const float cp = r.core[p];
    float cbound = shared_bound(r, c);
    const bool live = w + lane < count && r.k.low[p] < cbound;
    float q[P];
    load_point<P>(t.pts + int64_t(p) * P, q);
    float bd = live ? r.k.near_d[p] : -inf;
    int32_t bj = -1;
    warp_walk<P>(
        t, q, cp,
        [&] {
          const float thr = fminf(bd, cbound);
          return cp < thr || thr == inf ? thr : -inf;
        },
        [&](int node) { return r.node_comp[node] == c || !(r.node_core[node] < cbound); },
        [&](int node, bool want) {
          // another warp may have lowered the component's bound meanwhile
          cbound = fminf(cbound, shared_bound(r, c));
          const int32_t e = t.nend[node];
#pragma unroll 2
          for (int32_t s = t.nstart[node]; s < e; s++) {
            const float cs = r.core[s];
            const float d = fmaxf(fmaxf(rdist<P>(q, t.pts + int64_t(s) * P), cp), cs);
            if (want && d < bd && cs < cbound && r.comp[s] != c) {
              bd = d;
              bj = s;
              cbound = fminf(cbound, d);
            }
          }
        },
        r.status);
    if (live) keep_found(r, p, c, bd, bj, cbound);
  }
}

// One open point a warp: the two halves test a node's children, the lanes a
// leaf's points.
template <int P>
__device__ void search_one(const Round& r, int32_t count) {
  const TreeView& t = r.t;
  const int lane = threadIdx.x & 31;
  const float inf = __int_as_float(0x7f800000);
  for (;;) {
    int32_t w = 0;
    if (lane == 0) w = atomicAdd(r.next, 1);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (uint32_t(w) >= uint32_t(count)) break;
    const int32_t p = r.open[w];
    const int32_t c = r.comp[p];
    const float cp = r.core[p];
    float cbound = __shfl_sync(0xffffffffu, shared_bound(r, c), 0);
    float q[P];
    load_point<P>(t.pts + int64_t(p) * P, q);
    float bd = r.k.near_d[p];
    int32_t bj = -1;
    int sn[kMaxStack];
    float sl[kMaxStack];
    sn[0] = 0;
    sl[0] = 0.0f;
    int sp = 1;
    while (sp > 0) {
      const int node = sn[--sp];
      const float lb = sl[sp];
      const float thr = fminf(bd, cbound);
      // while nothing is known every node is open, boxes at infinity too
      if (!((lb < thr && cp < thr) || thr == inf)) continue;
      if (node >= t.first_leaf) {
        cbound = fminf(cbound, __shfl_sync(0xffffffffu, shared_bound(r, c), 0));
        const int32_t e = t.nend[node];
        for (int32_t s0 = t.nstart[node]; s0 < e; s0 += 32) {
          const int32_t s = s0 + lane;
          float d = inf;
          if (s < e && r.comp[s] != c && r.core[s] < cbound)
            d = fmaxf(fmaxf(rdist<P>(q, t.pts + int64_t(s) * P), cp), r.core[s]);
          const uint32_t low = __reduce_min_sync(0xffffffffu, __float_as_uint(d));
          if (__uint_as_float(low) < bd) {
            bd = __uint_as_float(low);
            bj = s0 + __ffs(__ballot_sync(0xffffffffu, __float_as_uint(d) == low)) - 1;
            cbound = fminf(cbound, bd);
          }
        }
        continue;
      }
      const int child = 2 * node + 1 + (lane >> 4);
      const float b = node_lower_bound<P>(q, t.lo + int64_t(child) * P, t.hi + int64_t(child) * P);
      const bool want = ((b < thr || thr == inf) && r.node_comp[child] != c && r.node_core[child] < cbound);
      const unsigned wants = __ballot_sync(0xffffffffu, want);
      const float bl = __shfl_sync(0xffffffffu, b, 0), br = __shfl_sync(0xffffffffu, b, 16);
      if (sp + 2 > kMaxStack) {  // cannot happen for the checked depths; stop rather than overrun
        atomicCAS(r.status, 0, 1);
        break;
      }
      // the nearer child is visited first (pushed last)
      const int near = bl <= br ? 0 : 1;
      if (wants >> (16 * (1 - near)) & 1u) {
        sn[sp] = 2 * node + 2 - near;
        sl[sp++] = near ? bl : br;
      }
      if (wants >> (16 * near) & 1u) {
        sn[sp] = 2 * node + 1 + near;
        sl[sp++] = near ? br : bl;
      }
    }
    if (lane == 0) keep_found(r, p, c, bd, bj, cbound);
  }
}

// A walk is a chain of dependent loads, so a round lasts as long as its
// longest walk unless there are warps enough to hide it: 32 points a warp left
// the 8,000 open points of the first round of 300,000 x 7 with two warps an SM
// and 8 cycles an instruction (4.2 ms), although a warp to each point issues
// twice the instructions.  Above `one_each` points (256 an SM) the shared walk
// has its warps and is the cheaper one (100,000 x 15, its second and third
// round: 9.3 and 5.9 ms, against 11.6 and 8.4 with a warp to each point).
// 300,000 x 7: five rounds 66 -> 8.1 ms (a stack per thread, every point of
// every component searched anew; the first two rounds now 0.5 and 0.3 ms).
template <int P>
__global__ void __launch_bounds__(128) boruvka_query_kernel(Round r, const int32_t* __restrict__ n_open,
                                                            int32_t one_each) {
  const int32_t count = *n_open;
  if (count > one_each) search_many<P>(r, count);
  else search_one<P>(r, count);
}

// Each component joins along its smallest (mr, position) candidate.
__global__ void boruvka_merge_kernel(int64_t n, const int32_t* __restrict__ comp,
                                     const unsigned long long* __restrict__ best, const int32_t* __restrict__ near_pos,
                                     int32_t* __restrict__ parent, int32_t* __restrict__ e_from,
                                     int32_t* __restrict__ e_to, float* __restrict__ e_w, int32_t* count, int64_t cap) {
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
    if (comp[p] != p) continue;  // one thread per component: its root
    const unsigned long long key = best[p];
    if (key == ~0ull) continue;
    const int32_t src = int32_t(uint32_t(key));
    const int32_t dst = near_pos[src];
    const float w = __uint_as_float(uint32_t(key >> 32));
    if (uf_unite(parent, src, dst)) add_edge(src, dst, w, e_from, e_to, e_w, count, cap);
  }
}

// (from, to, sqrt(mr)) rows in point indices; core distances in point order.
__global__ void emit_edges_kernel(int64_t m, const int32_t* __restrict__ order, const int32_t* __restrict__ e_from,
                                  const int32_t* __restrict__ e_to, const float* __restrict__ e_w,
                                  float* __restrict__ out) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += int64_t(gridDim.x) * blockDim.x) {
    out[3 * i] = float(order[e_from[i]]);
    out[3 * i + 1] = float(order[e_to[i]]);
    out[3 * i + 2] = __fsqrt_rn(e_w[i]);
  }
}

__global__ void scatter_core_kernel(int64_t n, const int32_t* __restrict__ order, const float* __restrict__ core_t,
                                    float* __restrict__ core) {
  for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x)
    core[order[p]] = core_t[p];
}

// ------------------------------------------------------------------ host

struct Arena {
  evoc_gpu_ctx* ctx;
  std::vector<void*> ptrs;
  explicit Arena(evoc_gpu_ctx* c) : ctx(c) {}
  ~Arena() {
    for (void* p : ptrs) cudaFreeAsync(p, ctx->stream);
  }
  template <class T>
  cudaError_t get(T** out, size_t count) {
    const cudaError_t e = pool_get(ctx, out, count);
    if (e == cudaSuccess) ptrs.push_back(*out);
    return e;
  }
};

template <int P>
int run(evoc_gpu_ctx* ctx, Arena& A, const float* d_x, int64_t n, int dim, int64_t ldx, int min_samples,
        float* d_edges, float* d_core, int64_t* n_edges) {
  cudaStream_t st = ctx->stream;
  const int sms = ctx->sms;
  // Node ranges, leaf flags (host): the reference's layout.
  int n_levels = int(std::floor(std::log2(double(std::max<int64_t>(n - 1, 1)) / double(kLeafSize)))) + 1;
  if (n_levels < 1) n_levels = 1;
  if (n_levels > 28) return fail(ctx, EVOC_ERR_ARG, "too many points for the tree (levels > 28)");
  const int n_nodes = (1 << n_levels) - 1;
  std::vector<int32_t> hs(static_cast<size_t>(n_nodes)), he(static_cast<size_t>(n_nodes));
  hs[0] = 0;
  he[0] = int32_t(n);
  for (int i = 0; i < n_nodes; i++) {
    if (2 * i + 2 < n_nodes) {
      const int32_t s = hs[size_t(i)], e = he[size_t(i)], mid = s + (e - s) / 2;
      hs[size_t(2 * i + 1)] = s;
      he[size_t(2 * i + 1)] = mid;
      hs[size_t(2 * i + 2)] = mid;
      he[size_t(2 * i + 2)] = e;
    }
  }
  float *Xp, *pts, *lo, *hi, *core, *node_core, *knn_d, *e_w;
  Known known;
  int32_t *order, *order2, *nstart, *nend, *split, *knn_pos, *parent, *comp, *node_comp, *arrived, *open,
      *e_from, *e_to, *counters;
  uint64_t *keys, *keys2;
  uint32_t* bound;
  unsigned long long* best;
  const int kq = min_samples > 1 ? min_samples + 1 : 2;
  const int64_t cap = n - 1;
  EVOC_TRY(A.get(&Xp, size_t(n) * P), "alloc points");
  EVOC_TRY(A.get(&pts, size_t(n) * P), "alloc points");
  EVOC_TRY(A.get(&lo, size_t(n_nodes) * P), "alloc bounds");
  EVOC_TRY(A.get(&hi, size_t(n_nodes) * P), "alloc bounds");
  EVOC_TRY(A.get(&order, size_t(n)), "alloc order");
  EVOC_TRY(A.get(&order2, size_t(n)), "alloc order");
  EVOC_TRY(A.get(&keys, size_t(n)), "alloc keys");
  EVOC_TRY(A.get(&keys2, size_t(n)), "alloc keys");
  EVOC_TRY(A.get(&nstart, size_t(n_nodes)), "alloc nodes");
  EVOC_TRY(A.get(&nend, size_t(n_nodes)), "alloc nodes");
  EVOC_TRY(A.get(&split, size_t(n_nodes)), "alloc nodes");
  EVOC_TRY(A.get(&node_comp, size_t(n_nodes)), "alloc nodes");
  EVOC_TRY(A.get(&core, size_t(n)), "alloc core");
  EVOC_TRY(A.get(&knn_pos, size_t(n) * kq), "alloc knn");
  EVOC_TRY(A.get(&knn_d, size_t(n) * kq), "alloc knn");
  EVOC_TRY(A.get(&parent, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&comp, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&node_core, size_t(n_nodes)), "alloc nodes");
  EVOC_TRY(A.get(&arrived, size_t(n_nodes)), "alloc nodes");
  EVOC_TRY(A.get(&open, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&known.low, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&known.near_pos, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&known.near_d, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&bound, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&best, size_t(n)), "alloc components");
  EVOC_TRY(A.get(&e_from, size_t(cap)), "alloc edges");
  EVOC_TRY(A.get(&e_to, size_t(cap)), "alloc edges");
  EVOC_TRY(A.get(&e_w, size_t(cap)), "alloc edges");
  EVOC_TRY(A.get(&counters, 16), "alloc counters");
  EVOC_TRY(cudaMemcpyAsync(nstart, hs.data(), hs.size() * 4, cudaMemcpyHostToDevice, st), "upload nodes");
  EVOC_TRY(cudaMemcpyAsync(nend, he.data(), he.size() * 4, cudaMemcpyHostToDevice, st), "upload nodes");
  EVOC_TRY(cudaMemsetAsync(counters, 0, 64, st), "clear counters");
  EVOC_TRY(cudaMemsetAsync(arrived, 0, size_t(n_nodes) * 4, st), "clear arrivals");
  int32_t* status = counters + 1;
  const int grid = sms * 8;
  {
    Stage s(ctx, "mst_tree");
    pad_points_kernel<<<grid, 256, 0, st>>>(d_x, n, dim, ldx, Xp, P);
    iota_kernel<<<grid, 256, 0, st>>>(order, n);
    EVOC_TRY(cudaGetLastError(), "pad points");
    ctx->launches += 2;
    size_t tmp_bytes = 0;
    EVOC_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, keys, keys2, order, order2, int(n), 0, 64, st),
             "sort size");
    void* tmp = nullptr;
    EVOC_TRY(A.get(reinterpret_cast<uint8_t**>(&tmp), tmp_bytes), "alloc sort");
    // levels above the subtrees that one block holds; none for the smallest sets
    int top = 0;
    while ((n + (int64_t(1) << top) - 1) >> top > Subtree<P>::kCap) top++;
    EVOC_TRY(cudaMemsetAsync(lo, 0xff, ((size_t(1) << top) - 1) * P * 4, st), "clear bounds");
    EVOC_TRY(cudaMemsetAsync(hi, 0, ((size_t(1) << top) - 1) * P * 4, st), "clear bounds");
    for (int l = 0; l < top; l++) {
      const int first = (1 << l) - 1, count = 1 << l;
      uint32_t *ulo = reinterpret_cast<uint32_t*>(lo), *uhi = reinterpret_cast<uint32_t*>(hi);
      const dim3 bgrid(unsigned(std::max(1, sms * 4 / count)), unsigned(std::min(count, sms * 4)));
      node_bounds_kernel<P><<<bgrid, 256, 0, st>>>(Xp, order, nstart, nend, first, count, ulo, uhi);
      node_split_kernel<P><<<(count + 127) / 128, 128, 0, st>>>(first, count, dim, ulo, uhi, split);
      split_keys_kernel<<<grid, 256, 0, st>>>(Xp, P, order, n, nstart, first, count, split, keys);
      EVOC_TRY(cudaGetLastError(), "split keys");
      int end_bit = 32;
      while ((1 << (end_bit - 32)) < count) end_bit++;
      EVOC_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys, keys2, order, order2, int(n), 0, end_bit, st),
               "split sort");
      std::swap(order, order2);
      ctx->launches += 4;
    }
    EVOC_TRY(cudaFuncSetAttribute(subtree_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(Subtree<P>::kSmem)),
             "subtree smem");
    subtree_kernel<P><<<1 << top, Subtree<P>::kThreads, Subtree<P>::kSmem, st>>>(Xp, order, nstart, nend, top,
                                                                                n_levels, dim, lo, hi, pts);
    EVOC_TRY(cudaGetLastError(), "subtrees");
    ctx->launches += 1;
  }
  const TreeView tv{n, n_nodes, order, pts, nstart, nend, n_nodes / 2, lo, hi};
  const int qgrid = int(std::min<int64_t>((n + 127) / 128, int64_t(sms) * 64));
  const int lgrid = (n_nodes - n_nodes / 2 + 127) / 128;
  {
    Stage s(ctx, "mst_core");
    if (kq <= 8) knn_kernel<P, 8><<<qgrid, 128, 0, st>>>(tv, kq, core, knn_pos, knn_d, status);
    else if (kq <= 16) knn_kernel<P, 16><<<qgrid, 128, 0, st>>>(tv, kq, core, knn_pos, knn_d, status);
    else knn_kernel<P, kMaxKnn><<<qgrid, 128, 0, st>>>(tv, kq, core, knn_pos, knn_d, status);
    EVOC_TRY(cudaGetLastError(), "core distances");
    ctx->launches += 1;
  }
  if (min_samples <= 1) EVOC_TRY(cudaMemsetAsync(core, 0, size_t(n) * 4, st), "zero core");
  int32_t *e_count = counters, *n_open = counters + 2, *next = counters + 3;
  {
    Stage s(ctx, "mst_init");
    iota_kernel<<<grid, 256, 0, st>>>(parent, n);
    knn_init_kernel<<<grid, 256, 0, st>>>(n, kq, core, knn_pos, knn_d, parent, e_from, e_to, e_w, e_count, cap);
    known_init_kernel<<<grid, 256, 0, st>>>(n, core, known);
    node_values_kernel<<<lgrid, 128, 0, st>>>(tv, nullptr, nullptr, core, node_core, arrived);
    EVOC_TRY(cudaGetLastError(), "knn init");
    ctx->launches += 4;
  }
  int32_t h[2] = {0, 0};
  Stage rounds(ctx, "mst_rounds");
  for (int round = 0;; round++) {
    const int32_t before = h[0];
    EVOC_TRY(cudaMemcpyAsync(h, counters, 8, cudaMemcpyDeviceToHost, st), "read edge count");
    EVOC_TRY(cudaStreamSynchronize(st), "mst round");
    if (h[1] != 0) return fail(ctx, EVOC_ERR_CUDA, "tree traversal stack overflow");
    if (h[0] >= cap) break;
    if (round > 0 && h[0] == before) return fail(ctx, EVOC_ERR_CUDA, "a Boruvka round joined no components");
    if (round > 64) return fail(ctx, EVOC_ERR_CUDA, "Boruvka did not converge");
    components_kernel<<<grid, 256, 0, st>>>(n, parent, comp, bound, best);
    node_values_kernel<<<lgrid, 128, 0, st>>>(tv, comp, node_comp, nullptr, nullptr, arrived);
    EVOC_TRY(cudaMemsetAsync(n_open, 0, 8, st), "clear counters");
    seed_kernel<<<grid, 256, 0, st>>>(n, kq, comp, core, knn_pos, knn_d, known, bound, best);
    open_points_kernel<<<grid, 256, 0, st>>>(n, comp, known.low, bound, open, n_open);
    const int query_grid = int(std::min<int64_t>((n + 3) / 4, int64_t(sms) * 8));
    const Round r{tv, core, comp, node_comp, node_core, open, next, known, bound, best, status};
    boruvka_query_kernel<P><<<query_grid, 128, 0, st>>>(r, n_open, sms * 256);
    boruvka_merge_kernel<<<grid, 256, 0, st>>>(n, comp, best, known.near_pos, parent, e_from, e_to, e_w, e_count, cap);
    EVOC_TRY(cudaGetLastError(), "boruvka round");
    ctx->launches += 6;
  }
  rounds.end();
  *n_edges = cap;
  emit_edges_kernel<<<grid, 256, 0, st>>>(cap, order, e_from, e_to, e_w, d_edges);
  if (d_core) scatter_core_kernel<<<grid, 256, 0, st>>>(n, order, core, d_core);
  EVOC_TRY(cudaGetLastError(), "emit edges");
  ctx->launches += d_core ? 2 : 1;
  return EVOC_OK;
}

int boruvka_impl(evoc_gpu_ctx* ctx, const float* data, int64_t n, int32_t dim, int32_t min_samples, int32_t on_dev,
                 float* out_edges, float* out_core, int64_t* n_edges) {
  if (!ctx) return EVOC_ERR_ARG;
  std::lock_guard<std::mutex> lock(ctx->mu);
  ctx->err.clear();
  ctx->n_stages = 0;
  ctx->launches = 0;
  if (n_edges) *n_edges = 0;
  if (n <= 0) return fail(ctx, EVOC_ERR_EMPTY, "no points");
  if (!data || (n > 1 && !out_edges)) return fail(ctx, EVOC_ERR_ARG, "null data or out_edges");
  if (dim < 1 || dim > 32) return fail(ctx, EVOC_ERR_ARG, "dim must be in 1..32");
  if (min_samples < 0 || min_samples + 1 > kMaxKnn) return fail(ctx, EVOC_ERR_ARG, "min_samples must be in 0..31");
  if (n >= (int64_t(1) << 31) - 1) return fail(ctx, EVOC_ERR_ARG, "n exceeds the int32 index range");
  const int kq = min_samples > 1 ? min_samples + 1 : 2;
  if (n < kq) return fail(ctx, EVOC_ERR_ARG, "need more than min_samples points (the core distance is undefined)");
  EVOC_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
  if (!ctx->lp_pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = ctx->device;
    EVOC_TRY(cudaMemPoolCreate(&ctx->lp_pool, &props), "memory pool");
    uint64_t keep = UINT64_MAX;
    EVOC_TRY(cudaMemPoolSetAttribute(ctx->lp_pool, cudaMemPoolAttrReleaseThreshold, &keep), "memory pool");
  }
  Stage total(ctx, "total");
  int rc = EVOC_OK;
  {
    Arena A(ctx);
    const float* d_x = data;
    float *d_edges = out_edges, *d_core = out_core;
    if (!on_dev) {
      float* xs;
      EVOC_TRY(A.get(&xs, size_t(n) * size_t(dim)), "alloc points");
      EVOC_TRY(cudaMemcpyAsync(xs, data, size_t(n) * size_t(dim) * 4, cudaMemcpyHostToDevice, ctx->stream),
               "upload points");
      d_x = xs;
      EVOC_TRY(A.get(&d_edges, size_t(std::max<int64_t>(n - 1, 1)) * 3), "alloc edges");
      d_core = nullptr;
      if (out_core) EVOC_TRY(A.get(&d_core, size_t(n)), "alloc core");
    }
    int64_t ne = 0;
    if (n == 1) {
      if (d_core) EVOC_TRY(cudaMemsetAsync(d_core, 0, 4, ctx->stream), "core");
    } else if (dim <= 4) {
      rc = run<4>(ctx, A, d_x, n, dim, dim, min_samples, d_edges, d_core, &ne);
    } else if (dim <= 8) {
      rc = run<8>(ctx, A, d_x, n, dim, dim, min_samples, d_edges, d_core, &ne);
    } else if (dim <= 16) {
      rc = run<16>(ctx, A, d_x, n, dim, dim, min_samples, d_edges, d_core, &ne);
    } else {
      rc = run<32>(ctx, A, d_x, n, dim, dim, min_samples, d_edges, d_core, &ne);
    }
    if (rc) return rc;
    if (!on_dev) {
      if (ne > 0)
        EVOC_TRY(cudaMemcpyAsync(out_edges, d_edges, size_t(ne) * 12, cudaMemcpyDeviceToHost, ctx->stream),
                 "download edges");
      if (out_core)
        EVOC_TRY(cudaMemcpyAsync(out_core, d_core, size_t(n) * 4, cudaMemcpyDeviceToHost, ctx->stream),
                 "download core");
    }
    if (n_edges) *n_edges = ne;
  }
  total.end();
  EVOC_TRY(cudaStreamSynchronize(ctx->stream), "boruvka");
  return EVOC_OK;
}

}  // namespace mst
}  // namespace evoc

extern "C" int evoc_gpu_boruvka_mst(evoc_gpu_ctx* ctx, const float* data, int64_t n, int32_t dim,
                                    int32_t min_samples, int32_t buffers_on_device, float* out_edges,
                                    float* out_core, int64_t* n_edges) {
  return evoc::mst::boruvka_impl(ctx, data, n, dim, min_samples, buffers_on_device, out_edges, out_core, n_edges);
}
