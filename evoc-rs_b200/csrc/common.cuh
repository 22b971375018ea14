// Shared device/host helpers for the evoc kNN-graph engine (sm_100a).
//
// Distance conventions follow the evoc-rs kNN path:
//   f32  raw = -dot if dot > 0 else f32::MIN_POSITIVE        src/fast_cosine.rs:33-45
//   i8   raw = -(dot_i32 as f32)                               src/nndescent/int8.rs:15-21
//   u8   raw = -(inter/union) (f32 div), 0.0 if union == 0     src/nndescent/uint8.rs:21-35
//   self raw = -1.0 (leaf-init rule)                           src/nndescent/float.rs:209-215
// Rows are ranked by the total order (raw, index) with f32 equality
// (-0.0 == +0.0), smallest first.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace evoc {

constexpr float kMinPositive = 1.17549435e-38f;  // f32::MIN_POSITIVE
constexpr float kHeapInf = 3.40282347e+38f;      // f32::MAX, heap.rs:8
constexpr uint64_t kKeyInf = ~0ull;

// Codes of a request's device status word (0 = ok).  1..3: a pipeline wait of
// the tensor-core scan ran out (producer, MMA issuer, epilogue); 4: a copy of
// the rerank did not arrive in time; 16, 17: a
// self-check found a malformed row order or a candidate index out of range
// and skipped it.
constexpr int kStatusBadOrder = 16;
constexpr int kStatusBadCandidate = 17;

// Order-preserving map f32 -> u32 (after folding -0.0 onto +0.0).
__device__ __forceinline__ uint32_t orderable(float f) {
  f = f + 0.0f;  // -0.0 + 0.0 == +0.0 under round-to-nearest
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float from_orderable(uint32_t o) {
  uint32_t u = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
  return __uint_as_float(u);
}

__device__ __forceinline__ uint64_t make_key(float raw, int32_t idx) {
  return (uint64_t(orderable(raw)) << 32) | uint32_t(idx);
}

__host__ __device__ __forceinline__ int32_t key_index(uint64_t key) { return int32_t(uint32_t(key)); }

__device__ __forceinline__ float raw_cosine(float dot) { return dot > 0.0f ? -dot : kMinPositive; }

__device__ __forceinline__ float raw_int8(int32_t dot) { return -__int2float_rn(dot); }

__device__ __forceinline__ float raw_jaccard(uint32_t inter, uint32_t uni) {
  return uni > 0 ? -__fdiv_rn(__uint2float_rn(inter), __uint2float_rn(uni)) : 0.0f;
}

// Ordering keys fold -0.0 onto +0.0.  An int8 dissimilarity of zero is
// -(0 as f32) = -0.0 in the reference, so the writer restores that sign.
__device__ __forceinline__ float int8_raw_from_key(float r) { return r == 0.0f ? -0.0f : r; }

// Distance transforms, src/knn.rs:156-187 (f64 log2 for f32/u8, f32 division for i8).
__device__ __forceinline__ float transform_raw(int dtype, float d) {
  if (dtype == 0) {
    if (d >= 0.0f) return 0.0f;
    double sim = double(-d);
    if (sim >= 1.0) return 0.0f;
    return float(fmax(-log2(sim), 0.0));
  } else if (dtype == 1) {
    return d >= 0.0f ? 0.0f : __fdiv_rn(1.0f, -d);
  } else {
    return d >= 0.0f ? 0.0f : float(-log2(double(-d)));
  }
}

// ---------------------------------------------------------------------------
// Thread-private candidate buffer: one owner thread per query row appends
// keys that beat its current threshold; when the buffer is full it keeps the
// k smallest (nth-element) and the k-th becomes the new threshold.  The final
// answer depends only on the set of keys offered, so it is deterministic.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void kswap(uint64_t* a, int i, int j) {
  uint64_t t = a[i];
  a[i] = a[j];
  a[j] = t;
}

// Rearranges buf[0..cnt) so that buf[0..k) hold the k smallest keys and
// buf[k-1] is the largest of them.  Requires 1 <= k <= cnt.
__device__ inline void nth_smallest(uint64_t* buf, int cnt, int k) {
  int lo = 0, hi = cnt - 1;
  const int target = k - 1;
  while (hi > lo) {
    int mid = lo + ((hi - lo) >> 1);
    // median-of-three pivot into buf[hi]
    if (buf[mid] < buf[lo]) kswap(buf, mid, lo);
    if (buf[hi] < buf[lo]) kswap(buf, hi, lo);
    if (buf[mid] < buf[hi]) kswap(buf, mid, hi);
    uint64_t pivot = buf[hi];
    int store = lo;
    for (int i = lo; i < hi; i++) {
      uint64_t v = buf[i];
      if (v < pivot) {
        buf[i] = buf[store];
        buf[store] = v;
        store++;
      }
    }
    kswap(buf, store, hi);
    if (store == target) return;
    if (store < target) lo = store + 1;
    else hi = store - 1;
  }
}

__device__ inline void sort_keys(uint64_t* buf, int cnt) {
  for (int i = 1; i < cnt; i++) {
    uint64_t v = buf[i];
    int j = i - 1;
    while (j >= 0 && buf[j] > v) {
      buf[j + 1] = buf[j];
      j--;
    }
    buf[j + 1] = v;
  }
}

struct RowTopK {
  uint64_t* buf;  // CAP entries, private to the owner thread
  int cnt;
  int k;
  int cap;
  uint64_t thr;   // keys >= thr cannot enter
  float thr_raw;  // raw part of thr (quick reject)

  __device__ __forceinline__ void init(uint64_t* b, int kk, int capacity) {
    buf = b;
    cnt = 0;
    k = kk;
    cap = capacity;
    thr = kKeyInf;
    thr_raw = __int_as_float(0x7f800000);  // +inf
  }

  __device__ __forceinline__ void compact() {
    nth_smallest(buf, cnt, k);
    cnt = k;
    thr = buf[k - 1];
    thr_raw = from_orderable(uint32_t(thr >> 32));
  }

  // Offer (raw, idx).  raw must not be NaN.
  __device__ __forceinline__ void offer(float raw, int32_t idx) {
    if (raw > thr_raw) return;
    uint64_t key = make_key(raw, idx);
    if (key >= thr) return;
    buf[cnt++] = key;
    if (cnt == cap) compact();
  }

  // Sorts and returns the number of valid entries (min(cnt, k)).
  __device__ __forceinline__ int finish() {
    if (cnt > k) compact();
    sort_keys(buf, cnt);
    return cnt;
  }
};

}  // namespace evoc

namespace evoc {

// ---------------------------------------------------------------------------
// Thread-private bounded max-heap of ordering keys (one owner thread per query
// row).  Holds the `cap` smallest keys offered so far; its root is the exact
// cap-th best, so it is also the admission threshold.  The storage may be
// shared memory (row stride chosen odd in 8-byte words, so the 32 owners of a
// warp touching the same slot hit distinct banks) or global memory.
// ---------------------------------------------------------------------------
struct KeyHeap {
  uint64_t* h;
  int size;
  int cap;

  __device__ __forceinline__ void init(uint64_t* storage, int capacity) {
    h = storage;
    size = 0;
    cap = capacity;
  }

  __device__ __forceinline__ uint64_t threshold() const { return size < cap ? kKeyInf : h[0]; }

  __device__ inline void sift_down(int e) {
    const uint64_t v = h[e];
    for (;;) {
      int c = 2 * e + 1;
      if (c >= cap) break;
      uint64_t cv = h[c];
      if (c + 1 < cap) {
        const uint64_t r = h[c + 1];
        if (r > cv) {
          cv = r;
          c++;
        }
      }
      if (cv <= v) break;
      h[e] = cv;
      e = c;
    }
    h[e] = v;
  }

  // Keys are unique (they embed the row index), so a strict compare suffices.
  __device__ inline void offer(uint64_t key) {
    if (size < cap) {
      h[size++] = key;
      if (size == cap)
        for (int e = cap / 2 - 1; e >= 0; e--) sift_down(e);
      return;
    }
    if (key >= h[0]) return;
    h[0] = key;
    sift_down(0);
  }

  // Sorts ascending in place (insertion sort; cap is small) and returns the count.
  __device__ inline int finish() {
    sort_keys(h, size);
    return size;
  }
};

// The same set kept as eight groups of slots with each group's largest key in
// registers.  An insert replaces the set's largest key, rescans that group's
// slots (independent loads) and takes the largest of the eight maxima: two
// short dependency chains instead of the heap's log2(cap) dependent
// load-compare-store steps down a path, at 20 registers more.  In the scan the
// inserts of a warp's 32 rows mostly run one after the other, so their latency
// paces it: 2,000 x 128 f32 rows at k = 15 scan in 205 us (heap: 287), 50,000 x
// 200 in 2.97 ms (3.59).  An insert reads cap / 8 slots, so the set is for few
// keys: takes_heap (tc_scan.cu) says where the line lies.  At most 65,535 slots.
struct KeySet {
  uint64_t* h;
  int size;
  int cap;
  int per;           // slots per group
  uint64_t top;      // largest key once size == cap
  uint32_t top_at;   // its slot, and its group in bits 16..
  uint64_t gm[8];    // each group's largest key
  uint32_t gs[8];    // and its slot

  __device__ __forceinline__ void init(uint64_t* storage, int capacity) {
    h = storage;
    size = 0;
    cap = capacity;
    per = (capacity + 7) >> 3;
    top = kKeyInf;
    top_at = 0;
#pragma unroll
    for (int g = 0; g < 8; g++) {
      gm[g] = 0;
      gs[g] = 0;
    }
  }

  __device__ __forceinline__ uint64_t threshold() const { return top; }

  // The largest key of a group and its slot.
  __device__ __forceinline__ void scan_group(int g, uint64_t& m, uint32_t& at) const {
    const int s0 = g * per, s1 = min(s0 + per, cap);
    m = 0;
    at = 0;
#pragma unroll 4
    for (int s = s0; s < s1; s++) {
      const uint64_t k = h[s];
      if (k >= m) {
        m = k;
        at = uint32_t(s);
      }
    }
  }

  __device__ __forceinline__ void find_top() {
    uint64_t m[4];
    uint32_t a[4];
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const bool up = gm[g + 4] > gm[g];
      m[g] = up ? gm[g + 4] : gm[g];
      a[g] = up ? gs[g + 4] | uint32_t(g + 4) << 16 : gs[g] | uint32_t(g) << 16;
    }
#pragma unroll
    for (int g = 0; g < 2; g++) {
      const bool up = m[g + 2] > m[g];
      m[g] = up ? m[g + 2] : m[g];
      a[g] = up ? a[g + 2] : a[g];
    }
    const bool up = m[1] > m[0];
    top = up ? m[1] : m[0];
    top_at = up ? a[1] : a[0];
  }

  __device__ inline void offer(uint64_t key) {
    if (size < cap) {
      h[size++] = key;
      if (size < cap) return;
#pragma unroll
      for (int g = 0; g < 8; g++) scan_group(g, gm[g], gs[g]);
      find_top();
      return;
    }
    if (key >= top) return;
    h[top_at & 0xffffu] = key;
    const int g = int(top_at >> 16);
    uint64_t m;
    uint32_t at;
    scan_group(g, m, at);
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (u == g) {
        gm[u] = m;
        gs[u] = at;
      }
    find_top();
  }

  // Sorts ascending in place (insertion sort; cap is small) and returns the count.
  __device__ inline int finish() {
    sort_keys(h, size);
    return size;
  }
};

}  // namespace evoc
