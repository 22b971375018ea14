// Fuzzy simplicial set from the kNN graph, on the device.
//
// Restates src/graph_construction.rs:16-248 and the SciPy-compatible sparse
// binops of src/csr_matmul.rs:62-150:
//   smooth_knn_dist       per row: rho = first distance > 0; sigma by 64 steps
//                         of bisection in f64 on sum_{j>=1} exp(-(d_j-rho)/sigma)
//                         = log2(k), tolerance 1e-5; floored at 1e-3 * mean(row)
//                         (rho > 0) or 1e-3 * mean(all distances) (rho == 0)
//   membership strengths  w = 0 for self, 1 when d - rho <= 0 or sigma == 0,
//                         else f32 exp(-(d - rho) / sigma)
//   fuzzy union           A + A^T - A o A^T, each element rounded in f32 in the
//                         order SciPy's row-wise merge rounds it, zeros dropped,
//                         rows sorted by column (canonical CSR)
//
// One thread owns one row for sigma/rho/membership, the rows of a block side
// by side in shared memory (a row's own 4-byte loads lie k words apart: 32
// sectors each, and the bisection reads the row ~25 times).  The transpose is
// a column count / scan / scatter / per-bucket sort of packed (row, value)
// words; the warp that sorts a bucket also counts the row of the union, and a
// second pass writes it, each entry's place found by binary search in the
// other side.  Rows of more than kRowMax neighbours take the thread-per-row
// forms that work in global memory.  300,000 rows at k = 30: see each kernel.
#include "common.cuh"
#include "kernels.h"

namespace evoc {

constexpr int kRowMax = 64;  // neighbours per row the shared-memory forms take

// ndarray's contiguous f32 sum (eight partial sums, then a short tail) divided
// by the element count in f32: the order that mean() rounds in.  Sequential by
// nature, so one thread runs it, and only when a row needs it.
__global__ void ndarray_mean_kernel(const float* __restrict__ x, int64_t len, const int* __restrict__ need_mean,
                                    float* __restrict__ mean_out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (*need_mean == 0) {
    *mean_out = 0.0f;
    return;
  }
  float p[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int64_t i = 0;
  for (; i + 8 <= len; i += 8)
#pragma unroll
    for (int j = 0; j < 8; j++) p[j] = __fadd_rn(p[j], x[i + j]);
  float acc = 0.0f;
  acc = __fadd_rn(acc, __fadd_rn(p[0], p[4]));
  acc = __fadd_rn(acc, __fadd_rn(p[1], p[5]));
  acc = __fadd_rn(acc, __fadd_rn(p[2], p[6]));
  acc = __fadd_rn(acc, __fadd_rn(p[3], p[7]));
  for (int64_t j = 0; i < len && j < 7; i++, j++) acc = __fadd_rn(acc, x[i]);
  *mean_out = len > 0 ? __fdiv_rn(acc, float(len)) : 0.0f;
}

// sigma of a row whose j-th distance is row(j): bisection, then the floor
// (mean_all: the mean of all distances, for rows without a positive one).
template <class Row>
__device__ __forceinline__ double row_sigma(Row row, int k, double r, double target, double tol, float mean_all) {
  double lo = 0.0, hi = __longlong_as_double(0x7ff0000000000000ll), mid = 1.0;
  for (int it = 0; it < 64; it++) {
    double ps = 0.0;
    for (int j = 1; j < k; j++) {
      const double d = double(row(j)) - r;
      ps += d > 0.0 ? exp(-(d / mid)) : 1.0;
    }
    if (fabs(ps - target) < tol) break;
    if (ps > target) {
      hi = mid;
      mid = (lo + hi) / 2.0;
    } else {
      lo = mid;
      if (isinf(hi)) mid *= 2.0;
      else mid = (lo + hi) / 2.0;
    }
  }
  double s = mid;
  if (r > 0.0) {
    double m = 0.0;
    for (int j = 0; j < k; j++) m += double(row(j));
    m /= double(k);
    const double fl = double(1e-3f) * m;
    if (s < fl) s = fl;
  } else {
    const double fl = double(1e-3f) * double(mean_all);
    if (s < fl) s = fl;
  }
  return s;
}

__device__ __forceinline__ float membership(int32_t c, int64_t i, float d, float rh, float sig) {
  if (c == int32_t(i)) return 0.0f;
  const float dr = __fsub_rn(d, rh);
  return (dr <= 0.0f || sig == 0.0f) ? 1.0f : expf(-__fdiv_rn(dr, sig));
}

// sigma/rho and the membership row of A (nonzero weights, sorted by column).
// Rows without a positive distance need the mean of all distances: the first
// launch leaves them out and sets *zero_rows, the second (`rest`) takes only
// them.  Bound by the f64 exponentials and quotients (about 25 steps x k a
// row).  300,000 x 30, with the flags and counts: 0.81 ms (rows read and
// sorted in global memory: 1.25).
constexpr int kFuzzyRows = 128;

__global__ void __launch_bounds__(kFuzzyRows)
fuzzy_rows_kernel(const int32_t* __restrict__ idx, const float* __restrict__ dist, int64_t n, int k, float n_neighbors,
                  bool rest, int* __restrict__ zero_rows, const float* __restrict__ mean_all,
                  float* __restrict__ sigma_out, float* __restrict__ rho_out, int32_t* __restrict__ a_cols,
                  float* __restrict__ a_vals, int32_t* __restrict__ a_cnt, int32_t* __restrict__ indeg) {
  extern __shared__ uint32_t words[];
  constexpr int S = kFuzzyRows + 1;  // words between a row's entries: the tile's reads and writes spread over the banks
  float* d = reinterpret_cast<float*>(words);            // distances; a row's first slots then take its values
  int32_t* c = reinterpret_cast<int32_t*>(words) + k * S;  // columns
  __shared__ int32_t cnts[kFuzzyRows];
  if (rest && *zero_rows == 0) return;
  const int t = threadIdx.x;
  const double target = log2(double(n_neighbors));
  const double tol = double(1e-5f);
  const int64_t tiles = (n + kFuzzyRows - 1) / kFuzzyRows;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t r0 = tile * kFuzzyRows;
    const int rows = int(min(int64_t(kFuzzyRows), n - r0));
    __syncthreads();
    for (int e = t; e < rows * k; e += kFuzzyRows) {
      const int r = e / k, j = e - r * k;
      d[j * S + r] = dist[r0 * k + e];
      c[j * S + r] = idx[r0 * k + e];
    }
    __syncthreads();
    int cnt = -1;  // not this launch's row
    if (t < rows) {
      const int64_t i = r0 + t;
      auto row = [&](int j) { return d[j * S + t]; };
      double r = 0.0;
      for (int j = 0; j < k; j++) {
        const double v = double(row(j));
        if (v > 0.0) {
          r = v;
          break;
        }
      }
      if (!rest && r == 0.0) *zero_rows = 1;
      if ((r == 0.0) == rest) {
        const float sig = float(row_sigma(row, k, r, target, tol, rest ? *mean_all : 0.0f)), rh = float(r);
        sigma_out[i] = sig;
        rho_out[i] = rh;
        cnt = 0;
        for (int j = 0; j < k; j++) {  // at most j entries kept before entry j: they never reach it
          const int32_t col = c[j * S + t];
          if (col == -1) continue;
          const float w = membership(col, i, row(j), rh, sig);
          if (w == 0.0f) continue;
          int p = cnt++;
          while (p > 0 && c[(p - 1) * S + t] > col) {  // insertion by column
            c[p * S + t] = c[(p - 1) * S + t];
            d[p * S + t] = d[(p - 1) * S + t];
            p--;
          }
          c[p * S + t] = col;
          d[p * S + t] = w;
        }
        a_cnt[i] = cnt;
      }
    }
    cnts[t] = cnt;
    __syncthreads();
    for (int e = t; e < rows * k; e += kFuzzyRows) {
      const int r = e / k, j = e - r * k;
      if (j < cnts[r]) {
        const int32_t col = c[j * S + r];
        a_cols[r0 * k + e] = col;
        a_vals[r0 * k + e] = d[j * S + r];
        atomicAdd(&indeg[col], 1);
      }
    }
  }
}

// The same for rows of more than kRowMax neighbours, in global memory.
__global__ void fuzzy_long_rows_kernel(const int32_t* __restrict__ idx, const float* __restrict__ dist, int64_t n,
                                       int k, float n_neighbors, bool rest, int* __restrict__ zero_rows,
                                       const float* __restrict__ mean_all, float* __restrict__ sigma_out,
                                       float* __restrict__ rho_out, int32_t* __restrict__ a_cols,
                                       float* __restrict__ a_vals, int32_t* __restrict__ a_cnt,
                                       int32_t* __restrict__ indeg) {
  if (rest && *zero_rows == 0) return;
  const double target = log2(double(n_neighbors));
  const double tol = double(1e-5f);
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const float* row = dist + i * k;
    double r = 0.0;
    for (int j = 0; j < k; j++) {
      const double v = double(row[j]);
      if (v > 0.0) {
        r = v;
        break;
      }
    }
    if (!rest && r == 0.0) *zero_rows = 1;
    if ((r == 0.0) != rest) continue;
    const float sig = float(row_sigma([&](int j) { return row[j]; }, k, r, target, tol, rest ? *mean_all : 0.0f));
    const float rh = float(r);
    sigma_out[i] = sig;
    rho_out[i] = rh;
    int32_t* cols = a_cols + i * k;  // the row's k output slots, filled in column order
    float* vals = a_vals + i * k;
    int cnt = 0;
    for (int j = 0; j < k; j++) {
      const int32_t c = idx[i * k + j];
      if (c == -1) continue;
      const float w = membership(c, i, row[j], rh, sig);
      if (w == 0.0f) continue;
      int p = cnt++;
      while (p > 0 && cols[p - 1] > c) {  // insertion by column
        cols[p] = cols[p - 1];
        vals[p] = vals[p - 1];
        p--;
      }
      cols[p] = c;
      vals[p] = w;
    }
    for (int t = 0; t < cnt; t++) atomicAdd(&indeg[cols[t]], 1);
    a_cnt[i] = cnt;
  }
}

// out[0] = 0, out[i+1] = cnt[0] + ... + cnt[i]: each block's sum goes to the
// last place of its stretch of `out`, one block turns those into running sums
// (their final values), and each block fills its stretch from the one before.
// (One block walking all counts: 0.35 ms at 300,000.)  Counts of one block take
// the last of the three launches alone, so that a small graph has no more than
// it had (1,000 x 5: 0.113 -> 0.093 ms).
constexpr int kScanItems = 4;
constexpr int kScanBlock = 1024 * kScanItems;
static_assert(kScanBlock == kScanOneBlock, "one launch for the counts of one block");

__device__ __forceinline__ int64_t scan_end(int64_t b, int64_t n) { return min((b + 1) * kScanBlock, n); }

// Inclusive sums over the block's 1,024 values; part: 32 words of shared memory.
__device__ __forceinline__ int64_t block_inclusive(int64_t v, int64_t* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t x = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += x;
  }
  if (lane == 31) part[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int64_t w = part[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t x = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += x;
    }
    part[lane] = w;
  }
  __syncthreads();
  return warp ? v + part[warp - 1] : v;
}

template <class T>
__global__ void __launch_bounds__(1024) count_sums_kernel(const T* __restrict__ cnt, int64_t n, int64_t* out) {
  __shared__ int64_t part[32];
  const int64_t b0 = int64_t(blockIdx.x) * kScanBlock;
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    const int64_t at = b0 + i * 1024 + threadIdx.x;
    if (at < n) s += cnt[at];
  }
  s = block_inclusive(s, part);
  if (threadIdx.x == 1023) out[scan_end(blockIdx.x, n)] = s;
}

__global__ void __launch_bounds__(1024) scan_sums_kernel(int64_t blocks, int64_t n, int64_t* out) {
  __shared__ int64_t part[32];
  __shared__ int64_t carry;
  if (threadIdx.x == 0) {
    carry = 0;
    out[0] = 0;
  }
  __syncthreads();
  for (int64_t b0 = 0; b0 < blocks; b0 += 1024) {
    const int64_t b = b0 + threadIdx.x;
    const int64_t s = block_inclusive(b < blocks ? out[scan_end(b, n)] : 0, part) + carry;
    if (b < blocks) out[scan_end(b, n)] = s;
    __syncthreads();
    if (threadIdx.x == 1023) carry = s;
    __syncthreads();
  }
}

template <class T>
__global__ void __launch_bounds__(1024) scan_counts_kernel(const T* __restrict__ cnt, int64_t n, int64_t* out) {
  __shared__ int64_t part[32];
  const int64_t b0 = int64_t(blockIdx.x) * kScanBlock, end = scan_end(blockIdx.x, n);
  const int64_t at = b0 + int64_t(threadIdx.x) * kScanItems;
  T v[kScanItems];
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    v[i] = at + i < end ? cnt[at + i] : 0;
    s += v[i];
  }
  const bool alone = gridDim.x == 1;  // then nobody else writes out[0] and out[n]
  if (alone && threadIdx.x == 0) out[0] = 0;
  int64_t run = block_inclusive(s, part) - s + (alone ? 0 : out[b0]);
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    run += v[i];
    if (at + i + 1 < end || (alone && at + i + 1 == end)) out[at + i + 1] = run;
  }
}

__device__ __forceinline__ uint64_t bucket_key(int32_t r, float v) {
  return (uint64_t(uint32_t(r)) << 32) | __float_as_uint(v);
}

// A thread per entry slot of A.
__global__ void scatter_transpose_kernel(const int32_t* __restrict__ a_cols, const float* __restrict__ a_vals,
                                         const int32_t* __restrict__ a_cnt, int64_t n, int k,
                                         const int64_t* __restrict__ colptr, int32_t* __restrict__ fill,
                                         uint64_t* __restrict__ at) {
  const int64_t total = n * k;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e / k;
    if (int(e - i * k) >= a_cnt[i]) continue;
    const int32_t c = a_cols[e];
    at[colptr[c] + atomicAdd(&fill[c], 1)] = bucket_key(int32_t(i), a_vals[e]);
  }
}

// Each column bucket of A^T sorted by row.  A row appears at most once in a
// column, so sorting the packed (row << 32 | value bits) keys sorts by row.
// Buckets hold k entries on average but hubs can hold thousands: a warp sorts
// each bucket of up to kWarpSort entries (bitonic, in registers up to 64, in
// the warp's shared-memory slice above); larger buckets are listed and sorted
// by a whole block each (kBlockSort entries in shared memory), and any larger
// still by one thread (Shell sort).
constexpr int kWarpSort = 1024;
constexpr int kBlockSort = 8192;
constexpr int kSortWarps = 4;

__device__ __forceinline__ void bitonic_shared(uint64_t* keys, int P, int tid, int nthreads, bool block) {
  for (int size = 2; size <= P; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = tid; i < (P >> 1); i += nthreads) {
        const int lo = 2 * stride * (i / stride) + (i % stride);
        const int hi = lo + stride;
        const bool up = (lo & size) == 0;
        const uint64_t a = keys[lo], b = keys[hi];
        if ((a > b) == up) {
          keys[lo] = b;
          keys[hi] = a;
        }
      }
      if (block) __syncthreads();
      else __syncwarp();
    }
  }
}

// 32 keys, one per lane, ascending (or descending) over the lanes.
__device__ __forceinline__ uint64_t sort32(uint64_t key, int lane, bool up) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const uint64_t other = __shfl_xor_sync(0xffffffffu, key, stride);
      const bool low = (lane & stride) == 0, dir = ((lane & size) == 0 || size == 32) == up;
      key = (low == dir) ? min(key, other) : max(key, other);
    }
  }
  return key;
}

// A bitonic run of 32 keys over the lanes, ascending.
__device__ __forceinline__ uint64_t merge32(uint64_t key, int lane) {
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    const uint64_t other = __shfl_xor_sync(0xffffffffu, key, stride);
    key = (lane & stride) == 0 ? min(key, other) : max(key, other);
  }
  return key;
}

__device__ void shell_sort_bucket(uint64_t* at, int64_t m) {
  const int gaps[] = {701, 301, 132, 57, 23, 10, 4, 1};
  for (int gi = 0; gi < 8; gi++) {
    const int64_t g = gaps[gi];
    if (g >= m) continue;
    for (int64_t a = g; a < m; a++) {
      const uint64_t key = at[a];
      int64_t b = a;
      while (b >= g && at[b - g] > key) {
        at[b] = at[b - g];
        b -= g;
      }
      at[b] = key;
    }
  }
}

// First of the m sorted keys whose row is not below r.
__device__ __forceinline__ int64_t lower_row(const uint64_t* at, int64_t m, int32_t r) {
  int64_t lo = 0, hi = m;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (int32_t(at[mid] >> 32) < r) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The place of A's entry j in bucket i of A^T.  Equal columns of a row pair up
// in order, as a two-pointer merge pairs them.
struct Partner {
  int64_t p;  // first key of the bucket not below the column
  int rank;   // equal columns before entry j
  bool hit;   // the bucket holds entry p + rank of the same column
};
__device__ __forceinline__ Partner partner(const int32_t* cols, int j, const uint64_t* at, int64_t m) {
  Partner o;
  const int32_t col = cols[j];
  o.rank = 0;
  while (o.rank < j && cols[j - o.rank - 1] == col) o.rank++;
  o.p = lower_row(at, m, col);
  o.hit = o.p + o.rank < m && int32_t(at[o.p + o.rank] >> 32) == col;
  return o;
}

// Entries of row c of A (cnt of them) that have a partner in bucket c (m sorted keys).
__device__ __forceinline__ int common_columns(const int32_t* cols, int cnt, const uint64_t* at, int64_t m, int tid,
                                              int nthreads) {
  int both = 0;
  for (int j = tid; j < cnt; j += nthreads) both += partner(cols, j, at, m).hit ? 1 : 0;
  return both;
}

// A warp per bucket: sorts it and counts row c of the union.  With the prefix
// sums and the scatter, 300,000 x 30: 0.64 ms (every bucket sorted in shared
// memory, rows counted by a thread each, one block's prefix sums: 1.65).  No entry of the
// union is zero: weights are in (0, 1], and the rounded a + b is above the
// rounded a b.
__global__ void __launch_bounds__(kSortWarps * 32)
sort_buckets_warp_kernel(const int64_t* __restrict__ colptr, int64_t n, uint64_t* at, const int32_t* __restrict__ a_cols,
                         const int32_t* __restrict__ a_cnt, int k, int32_t* __restrict__ row_cnt,
                         int32_t* __restrict__ big, int32_t* __restrict__ n_big) {
  __shared__ uint64_t slice[kSortWarps][kWarpSort];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* keys = slice[warp];
  const int64_t wstride = int64_t(gridDim.x) * kSortWarps;
  for (int64_t c = int64_t(blockIdx.x) * kSortWarps + warp; c < n; c += wstride) {
    const int64_t s = colptr[c], m = colptr[c + 1] - s;
    uint64_t* b = at + s;
    if (m > kWarpSort) {
      if (lane == 0) big[atomicAdd(n_big, 1)] = int32_t(c);
      continue;
    }
    __syncwarp();
    if (m <= 64) {
      uint64_t x = lane < m ? b[lane] : ~0ull;
      if (m > 32) {
        uint64_t y = lane + 32 < m ? b[lane + 32] : ~0ull;
        x = sort32(x, lane, true);
        y = sort32(y, lane, false);
        const uint64_t l = min(x, y), h = max(x, y);
        x = merge32(l, lane);
        y = merge32(h, lane);
        if (lane + 32 < m) b[lane + 32] = y;
        keys[lane + 32] = y;
      } else if (m > 1) {
        x = sort32(x, lane, true);
      }
      if (lane < m) b[lane] = x;
      keys[lane] = x;
      __syncwarp();
    } else {
      int P = 128;
      while (P < m) P <<= 1;
      for (int i = lane; i < P; i += 32) keys[i] = i < m ? b[i] : ~0ull;
      __syncwarp();
      bitonic_shared(keys, P, lane, 32, false);
      for (int i = lane; i < m; i += 32) b[i] = keys[i];
    }
    const int cnt = a_cnt[c];
    const int both = __reduce_add_sync(0xffffffffu, common_columns(a_cols + c * k, cnt, keys, m, lane, 32));
    if (lane == 0) row_cnt[c] = cnt + int(m) - both;
  }
}

__global__ void sort_buckets_big_kernel(const int64_t* __restrict__ colptr, uint64_t* at,
                                        const int32_t* __restrict__ a_cols, const int32_t* __restrict__ a_cnt, int k,
                                        int32_t* __restrict__ row_cnt, const int32_t* __restrict__ big,
                                        const int32_t* __restrict__ n_big) {
  extern __shared__ uint64_t keys[];
  __shared__ int total;
  for (int b = blockIdx.x; b < *n_big; b += gridDim.x) {
    const int64_t c = big[b];
    const int64_t s = colptr[c], m = colptr[c + 1] - s;
    uint64_t* v = at + s;
    if (threadIdx.x == 0) total = 0;
    if (m > kBlockSort) {  // beyond a block's shared memory: one thread
      if (threadIdx.x == 0) shell_sort_bucket(v, m);
      __syncthreads();
    } else {
      int P = 1;
      while (P < m) P <<= 1;
      for (int i = threadIdx.x; i < P; i += blockDim.x) keys[i] = i < m ? v[i] : ~0ull;
      __syncthreads();
      bitonic_shared(keys, P, threadIdx.x, blockDim.x, true);
      for (int i = threadIdx.x; i < m; i += blockDim.x) v[i] = keys[i];
      __syncthreads();
    }
    const int both = common_columns(a_cols + c * k, a_cnt[c], v, m, threadIdx.x, blockDim.x);
    if (both) atomicAdd(&total, both);
    __syncthreads();
    if (threadIdx.x == 0) row_cnt[c] = a_cnt[c] + int(m) - total;
    __syncthreads();
  }
}

// Row i of (A + A^T) - (A o A^T), a warp per row: s = a + b (missing side is
// 0.0), p = a * b only where both exist, result s - p, in SciPy's rounding.
// An entry's place is its own index, plus the smaller columns of the other
// side, less the pairs of smaller columns.  300,000 x 30: 0.21 ms (a thread
// walking both sides of a row: 0.45).
constexpr int kUnionWarps = 8;

__global__ void __launch_bounds__(kUnionWarps * 32)
union_rows_kernel(int64_t n, int k, const int32_t* __restrict__ a_cols, const float* __restrict__ a_vals,
                  const int32_t* __restrict__ a_cnt, const int64_t* __restrict__ colptr,
                  const uint64_t* __restrict__ at, const int64_t* __restrict__ indptr, int32_t* __restrict__ indices,
                  float* __restrict__ data) {
  const int lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  const int64_t warps = int64_t(gridDim.x) * kUnionWarps;
  for (int64_t i = int64_t(blockIdx.x) * kUnionWarps + (threadIdx.x >> 5); i < n; i += warps) {
    const int32_t* cols = a_cols + i * k;
    const float* vals = a_vals + i * k;
    const int ca = a_cnt[i];
    const int64_t s = colptr[i], m = colptr[i + 1] - s;
    const uint64_t* b = at + s;
    int32_t* oc = indices + indptr[i];
    float* ov = data + indptr[i];
    int both = 0;  // columns of both sides in the chunks before
    for (int j0 = 0; j0 < ca; j0 += 32) {  // A's entries, with their partners
      const int j = j0 + lane;
      Partner q{0, 0, false};
      if (j < ca) q = partner(cols, j, b, m);
      const uint32_t who = __ballot_sync(0xffffffffu, q.hit);
      if (j < ca) {
        const int32_t col = cols[j];
        int pairs = q.rank;  // pairs of the same column before entry j
        if (!q.hit) {
          for (pairs = 0; q.p + pairs < m && int32_t(b[q.p + pairs] >> 32) == col;) pairs++;
        }
        const float va = vals[j], vb = q.hit ? __uint_as_float(uint32_t(b[q.p + q.rank])) : 0.0f;
        const int64_t o = j + q.p - (both + __popc(who & below) - pairs);
        oc[o] = col;
        ov[o] = __fsub_rn(__fadd_rn(va, vb), q.hit ? __fmul_rn(va, vb) : 0.0f);
      }
      both += __popc(who);
    }
    both = 0;
    for (int64_t j0 = 0; j0 < m; j0 += 32) {  // A^T's entries without one
      const int64_t j = j0 + lane;
      uint64_t key = 0;
      int p = 0, pairs = 0;  // smaller columns of A; pairs of the same column before entry j
      bool hit = false;
      if (j < m) {
        key = b[j];
        const int32_t col = int32_t(key >> 32);
        int hi = ca;
        while (p < hi) {
          const int mid = (p + hi) >> 1;
          if (cols[mid] < col) p = mid + 1;
          else hi = mid;
        }
        int64_t rank = 0;
        while (rank < j && int32_t(b[j - rank - 1] >> 32) == col) rank++;
        while (pairs < rank && p + pairs < ca && cols[p + pairs] == col) pairs++;
        hit = pairs == rank && p + pairs < ca && cols[p + pairs] == col;
      }
      const uint32_t who = __ballot_sync(0xffffffffu, hit);
      if (j < m && !hit) {
        const int64_t o = j + p - (both + __popc(who & below) - pairs);
        oc[o] = int32_t(key >> 32);
        ov[o] = __fsub_rn(__fadd_rn(0.0f, __uint_as_float(uint32_t(key))), 0.0f);
      }
      both += __popc(who);
    }
  }
}

// Without the transpose: the rows of A as they are.
__global__ void copy_rows_csr_kernel(int64_t n, int k, const int32_t* __restrict__ a_cols,
                                     const float* __restrict__ a_vals, const int32_t* __restrict__ a_cnt,
                                     const int64_t* __restrict__ indptr, int32_t* __restrict__ indices,
                                     float* __restrict__ data) {
  const int64_t total = n * k;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e / k;
    const int t = int(e - i * k);
    if (t < a_cnt[i]) {
      indices[indptr[i] + t] = a_cols[e];
      data[indptr[i] + t] = a_vals[e];
    }
  }
}

template <class T>
static cudaError_t scan_counts(const T* cnt, int64_t n, int64_t* out, cudaStream_t stream) {
  if (n <= 0) return cudaMemsetAsync(out, 0, sizeof(int64_t), stream);
  const unsigned blocks = unsigned((n + kScanBlock - 1) / kScanBlock);
  if (blocks > 1) {
    count_sums_kernel<<<blocks, 1024, 0, stream>>>(cnt, n, out);
    scan_sums_kernel<<<1, 1024, 0, stream>>>(blocks, n, out);
  }
  scan_counts_kernel<<<blocks, 1024, 0, stream>>>(cnt, n, out);
  return cudaGetLastError();
}

cudaError_t launch_scan_counts(const int32_t* cnt, int64_t n, int64_t* out, cudaStream_t stream) {
  return scan_counts(cnt, n, out, stream);
}

cudaError_t launch_scan_counts(const int64_t* cnt, int64_t n, int64_t* out, cudaStream_t stream) {
  return scan_counts(cnt, n, out, stream);
}

cudaError_t launch_smooth_and_membership(const int32_t* idx, const float* dist, int64_t n, int k, float n_neighbors,
                                         const FuzzyWork& w, float* sigma, float* rho, int sms, cudaStream_t stream) {
  if (k < 1) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(w.flags, 0, 2 * sizeof(int), stream);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(w.indeg, 0, size_t(n) * sizeof(int32_t), stream);
  if (e != cudaSuccess) return e;
  const size_t smem = size_t(2) * k * (kFuzzyRows + 1) * 4;
  if (k <= kRowMax) {
    e = cudaFuncSetAttribute(fuzzy_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * kRowMax * (kFuzzyRows + 1) * 4);
    if (e != cudaSuccess) return e;
  }
  for (int rest = 0; rest < 2; rest++) {
    if (rest) ndarray_mean_kernel<<<1, 32, 0, stream>>>(dist, n * int64_t(k), w.flags, w.mean);
    if (k <= kRowMax)
      fuzzy_rows_kernel<<<unsigned(std::min<int64_t>((n + kFuzzyRows - 1) / kFuzzyRows, int64_t(sms) * 32)),
                          kFuzzyRows, smem, stream>>>(idx, dist, n, k, n_neighbors, rest != 0, w.flags, w.mean, sigma,
                                                      rho, w.a_cols, w.a_vals, w.a_cnt, w.indeg);
    else
      fuzzy_long_rows_kernel<<<sms * 8, 128, 0, stream>>>(idx, dist, n, k, n_neighbors, rest != 0, w.flags, w.mean,
                                                          sigma, rho, w.a_cols, w.a_vals, w.a_cnt, w.indeg);
  }
  return cudaGetLastError();
}

cudaError_t launch_fuzzy_union_count(int64_t n, int k, int symmetrize, const FuzzyWork& w, int64_t* indptr, int sms,
                                     cudaStream_t stream) {
  if (!symmetrize) return launch_scan_counts(w.a_cnt, n, indptr, stream);
  cudaError_t e = launch_scan_counts(w.indeg, n, w.colptr, stream);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(w.fill, 0, size_t(n) * sizeof(int32_t), stream);
  if (e != cudaSuccess) return e;
  scatter_transpose_kernel<<<sms * 16, 256, 0, stream>>>(w.a_cols, w.a_vals, w.a_cnt, n, k, w.colptr, w.fill, w.at);
  e = cudaMemsetAsync(w.n_big, 0, sizeof(int32_t), stream);
  if (e != cudaSuccess) return e;
  sort_buckets_warp_kernel<<<sms * 16, kSortWarps * 32, 0, stream>>>(w.colptr, n, w.at, w.a_cols, w.a_cnt, k,
                                                                     w.row_cnt, w.big, w.n_big);
  e = cudaFuncSetAttribute(sort_buckets_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           int(kBlockSort * sizeof(uint64_t)));
  if (e != cudaSuccess) return e;
  sort_buckets_big_kernel<<<sms, 1024, kBlockSort * sizeof(uint64_t), stream>>>(w.colptr, w.at, w.a_cols, w.a_cnt, k,
                                                                                w.row_cnt, w.big, w.n_big);
  return launch_scan_counts(w.row_cnt, n, indptr, stream);
}

cudaError_t launch_fuzzy_union_write(int64_t n, int k, int symmetrize, const FuzzyWork& w, const int64_t* indptr,
                                     int32_t* indices, float* data, int sms, cudaStream_t stream) {
  if (symmetrize)
    union_rows_kernel<<<unsigned(std::min<int64_t>((n + kUnionWarps - 1) / kUnionWarps, int64_t(sms) * 64)),
                        kUnionWarps * 32, 0, stream>>>(n, k, w.a_cols, w.a_vals, w.a_cnt, w.colptr, w.at, indptr,
                                                       indices, data);
  else
    copy_rows_csr_kernel<<<sms * 16, 256, 0, stream>>>(n, k, w.a_cols, w.a_vals, w.a_cnt, indptr, indices, data);
  return cudaGetLastError();
}

}  // namespace evoc
