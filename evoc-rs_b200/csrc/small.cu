// Exact search of small sets: the scores written out by one product, then each
// row's nearest keys selected from them.
//
// The scan walks all key tiles in one CTA per 128 query rows and keeps keys
// as it goes.  A set of 2,000 rows then occupies 16 of 148 SMs, and most of
// its time goes into the first keys of every row's set.  Up to kSmallRows rows
// the tensor cores write the scores, a tile per CTA and at most kScoreBytes at
// a time so that they stay in L2, and a warp per row selects: 256 sampled
// scores give a bound that a few times `keep` keys reach, one pass over the
// row lists these, and bisection on the list's values finds the cut, ties by
// row index.  Where the list comes out too short or too long (many equal
// scores), the bisection goes over the whole row.  The kept sets are those of
// the scan.  Bound by the pass over the scores (about 10 instructions per 32,
// and L2 latency).  Against the scan: 2,000 x 128 rows f32 at k = 15 45 us
// (205), the whole call 165 us (316); 4,000 x 128 int8 122 us (198), 5,000 189
// (205), 6,500 294 (225), which is where kSmallRows comes from.  The scan's
// cost grows with the kept keys, this one's does not: int8 calls at k = 5 take
// 90 us (114) at 3,000 rows and 184 (129) at 4,900, where k = 40 takes 199
// (466), so int8 (whose calls are little more than the scan) has its line at
// 2,600 + 180 keep rows up to kSmallRows.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace evoc {

namespace {
constexpr int kWarps = 8;
constexpr uint32_t kNoKey = 0xffffffffu;   // ordering word of no column
constexpr uint32_t kLastKey = kNoKey - 1;  // no score's word is above it

template <int MODE>
__device__ __forceinline__ float score_raw(uint32_t bits, int32_t pa, int32_t pb) {
  if (MODE == kScanJaccard) {
    const int32_t inter = int32_t(bits), uni = pa + pb - inter;
    return uni > 0 ? -__fdiv_rn(__int2float_rn(inter), __int2float_rn(uni)) : 0.0f;
  }
  return MODE == kScanInt8 ? -__int2float_rn(int32_t(bits)) : raw_cosine(__uint_as_float(bits));
}

// Ordering word of a score; a NaN (of a row that holds one) passes no threshold of the scan and is
// never kept.
template <int MODE>
__device__ __forceinline__ uint32_t score_word(uint32_t bits, bool self, int32_t pa, int32_t pb) {
  const uint32_t word = orderable(self ? -1.0f : score_raw<MODE>(bits, pa, pb));
  return MODE == kScanHalf && !self && isnan(__uint_as_float(bits)) ? kNoKey : word;
}
}  // namespace

constexpr int kSample = 8;                    // sampled scores per lane
constexpr int kAhead = 8;                     // scores a lane loads ahead
constexpr size_t kScoreBytes = size_t(64) << 20;

template <int MODE>
__global__ void __launch_bounds__(kWarps * 32)
select_scores_kernel(const uint32_t* __restrict__ S, int64_t ld, int n_q, int n_k, int q_row0, int keep, int cap,
                     int final_mode, int dtype, const int32_t* __restrict__ pc, int32_t* __restrict__ out_idx,
                     float* __restrict__ out_raw, float* __restrict__ out_dist, float* __restrict__ out_bound,
                     const int* status) {
  extern __shared__ uint64_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (*reinterpret_cast<const volatile int*>(status) != 0) return;  // the scores are not complete
  uint64_t* list = smem + int64_t(warp) * (cap + keep);
  uint64_t* keys = list + cap;
  const uint32_t below = (1u << lane) - 1u;
  const int want = min(keep, n_k);
  for (int q = blockIdx.x * kWarps + warp; q < n_q; q += gridDim.x * kWarps) {
    const uint32_t* s = S + int64_t(q) * ld;
    const int self = q_row0 + q;
    const int32_t pa = MODE == kScanJaccard ? pc[self] : 0;
    auto key_of = [&](int c) {  // ordering word of column c
      return score_word<MODE>(s[c], c == self, pa, MODE == kScanJaccard ? pc[c] : 0);
    };
    // a bound that about 2.5 keep keys reach, and six sampled ones more for the spread
    uint32_t bound = kLastKey;
    if (n_k > 256) {
      uint32_t v[kSample];
      uint32_t lo = kNoKey, hi = 0u;
#pragma unroll
      for (int i = 0; i < kSample; i++) {
        v[i] = key_of(int((int64_t(i * 32 + lane) * n_k) >> 8));
        lo = min(lo, v[i]);
        hi = max(hi, v[i]);
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      const int rank = min(int(int64_t(640) * keep / n_k) + 6, 256);
      int c = 256;
      while (c > rank && lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        int t = 0;
#pragma unroll
        for (int i = 0; i < kSample; i++) t += v[i] <= mid ? 1 : 0;
        t = __reduce_add_sync(0xffffffffu, t);
        if (t >= rank) {
          hi = mid;
          c = t;
        } else {
          lo = mid + 1;
        }
      }
      bound = min(hi, kLastKey);
    }
    int m = 0;  // keys within the bound; the first `cap` are listed, in row order
    uint32_t lo = kNoKey, hi = 0u;
    for (int b = 0; b < n_k; b += 32 * kAhead) {
      uint32_t v[kAhead];
      int32_t pb[MODE == kScanJaccard ? kAhead : 1];
#pragma unroll
      for (int i = 0; i < kAhead; i++) {  // all loads before the first use
        const int c = min(b + 32 * i + lane, n_k - 1);
        v[i] = s[c];
        if (MODE == kScanJaccard) pb[i] = pc[c];
      }
#pragma unroll
      for (int i = 0; i < kAhead; i++) {
        const int c = b + 32 * i + lane;
        const uint32_t o =
            c < n_k ? score_word<MODE>(v[i], c == self, pa, pb[MODE == kScanJaccard ? i : 0]) : kNoKey;
        const bool in = o <= bound;
        const uint32_t who = __ballot_sync(0xffffffffu, in);
        const int at = m + __popc(who & below);
        if (in && at < cap) list[at] = (uint64_t(o) << 32) | uint32_t(c);
        lo = min(lo, o);
        hi = max(hi, in ? o : 0u);
        m += __popc(who);
      }
    }
    __syncwarp();
    const bool listed = m >= want && m <= cap;
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = listed ? __reduce_max_sync(0xffffffffu, hi) : kLastKey;
    const int len = listed ? m : n_k;  // what the cut is searched in
    auto word = [&](int i) { return listed ? uint32_t(list[i] >> 32) : key_of(i); };
    int upto = len;  // words <= hi
    while (upto > want && lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      int c = 0;
#pragma unroll 4
      for (int i = lane; i < len; i += 32) c += word(i) <= mid ? 1 : 0;
      c = __reduce_add_sync(0xffffffffu, c);
      if (c >= want) {
        hi = mid;
        upto = c;
      } else {
        lo = mid + 1;
      }
    }
    int ties = 0x7fffffff;  // words equal to hi that stay: all, or what the smaller ones leave room for
    if (upto > want) {
      int c = 0;
      for (int i = lane; i < len; i += 32) c += word(i) < hi ? 1 : 0;
      ties = want - __reduce_add_sync(0xffffffffu, c);
    }
    int out = 0, seen = 0;
    uint32_t worst = 0u;
    for (int b = 0; b < len; b += 32) {  // in row order, so the smaller indices of a tie come first
      const int i = b + lane;
      const uint32_t o = i < len ? word(i) : kNoKey;
      const uint32_t equal = __ballot_sync(0xffffffffu, o == hi);
      const bool in = o < hi || (o == hi && seen + __popc(equal & below) < ties);
      const uint32_t who = __ballot_sync(0xffffffffu, in);
      if (in) {
        keys[out + __popc(who & below)] = listed ? list[i] : (uint64_t(o) << 32) | uint32_t(i);
        worst = max(worst, o);
      }
      out += __popc(who);
      seen += __popc(equal);
    }
    __syncwarp();
    worst = __reduce_max_sync(0xffffffffu, worst);
    for (int j = lane; j < keep; j += 32) {
      float raw = kHeapInf;
      int32_t idx = -1;
      int at = j;
      if (j < out) {
        const uint64_t key = keys[j];
        raw = from_orderable(uint32_t(key >> 32));
        idx = key_index(key);
        if (final_mode) {  // the key's rank
          at = 0;
          for (int t = 0; t < out; t++) at += keys[t] < key ? 1 : 0;
        }
        // keys fold -0.0 onto +0.0: an int8 zero dot is -0.0, a Jaccard zero +0.0 only for two empty rows
        if (MODE == kScanInt8) raw = int8_raw_from_key(raw);
        if (MODE == kScanJaccard && raw == 0.0f) raw = (pa + pc[idx] == 0) ? 0.0f : -0.0f;
      }
      const int64_t o = int64_t(q) * keep + at;
      out_idx[o] = idx;
      if (out_raw) out_raw[o] = raw;
      if (final_mode && out_dist) out_dist[o] = transform_raw(dtype, raw);
    }
    if (out_bound && lane == 0) out_bound[q] = out == keep ? from_orderable(worst) : kHeapInf;
    __syncwarp();
  }
}

namespace {
int list_cap(int64_t n_k, int keep) { return int(std::min<int64_t>((n_k + 31) / 32 * 32, keep <= 96 ? 1024 : 2048)); }

// Query rows whose scores are written at a time: a multiple of 128.
int64_t score_rows(int64_t n_q, int64_t n_k) {
  const int64_t fit = std::max<int64_t>(int64_t(kScoreBytes) / (padded_rows(n_k) * 4) / 128 * 128, 128);
  return std::min<int64_t>(fit, (n_q + 127) / 128 * 128);
}
}  // namespace

bool small_scan_feasible(int mode, int64_t n_k, int keep) {
  return n_k <= kSmallRows && keep <= 256 && (mode != kScanInt8 || n_k <= 2600 + 180 * int64_t(keep));
}

size_t small_scan_bytes(int64_t n_q, int64_t n_k) {
  return size_t(score_rows(n_q, n_k)) * size_t(padded_rows(n_k)) * 4;
}

int small_scan_launches(int64_t n_q, int64_t n_k) {
  const int64_t step = score_rows(n_q, n_k);
  return 2 * int((n_q + step - 1) / step);
}

cudaError_t launch_small_scan(int mode, const void* X, int64_t rows_mem, int64_t n, int64_t q_row0, int64_t n_q,
                              int64_t row_bytes, int keep, int final_mode, int dtype, void* scores, int32_t* out_idx,
                              float* out_raw, float* out_dist, float* out_bound, int* status, uint64_t timeout_ns,
                              const int32_t* pc, int half_type, int sms, cudaStream_t stream) {
  if (!small_scan_feasible(mode, n, keep) || rows_mem < n || q_row0 < 0 || q_row0 + n_q > n || n_q < 1 || !status ||
      (mode == kScanJaccard && !pc))
    return cudaErrorInvalidValue;
  const int64_t ld = padded_rows(n), step = score_rows(n_q, n);
  const int cap = list_cap(n, keep);
  const size_t smem = size_t(kWarps) * size_t(cap + keep) * 8;
  cudaError_t e = cudaSuccess;
  for (int64_t q = 0; q < n_q; q += step) {
    const int64_t rows = std::min(step, n_q - q), r0 = q_row0 + q;
    e = launch_centre_products(mode == kScanHalf ? kScanHalf : kScanInt8,
                               static_cast<const uint8_t*>(X) + r0 * row_bytes, rows_mem - r0, rows, X, ld, row_bytes,
                               half_type, nullptr, scores, ld, status, timeout_ns, sms, stream, true);
    if (e != cudaSuccess) return e;
    const int64_t blocks = (rows + kWarps - 1) / kWarps, o = q * keep;
    auto go = [&](auto kern) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return e;
      kern<<<unsigned(std::min<int64_t>(blocks, int64_t(sms) * 8)), kWarps * 32, smem, stream>>>(
          static_cast<const uint32_t*>(scores), ld, int(rows), int(n), int(r0), keep, cap, final_mode, dtype, pc,
          out_idx + o, out_raw ? out_raw + o : nullptr, out_dist ? out_dist + o : nullptr,
          out_bound ? out_bound + q : nullptr, status);
      return cudaGetLastError();
    };
    e = mode == kScanHalf   ? go(select_scores_kernel<kScanHalf>)
        : mode == kScanInt8 ? go(select_scores_kernel<kScanInt8>)
                            : go(select_scores_kernel<kScanJaccard>);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace evoc
