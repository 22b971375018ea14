// Input preparation on the device.
//
// prepare_float (src/knn.rs:78-113): if any row's L2 norm differs from 1 by
// more than 1e-5, every row is divided by its norm (a zero norm divides by 1).
// The norm is the serial f32 sum of squares followed by sqrt, exactly as the
// reference rounds it: each product and each partial sum is rounded on its
// own (no FMA contraction), sqrt and division are IEEE.
//
// One pass reads the caller's rows and writes everything the search wants of
// them: the padded f32 rows, the norms, the 16-bit rows and their certificate
// norms, taking the rows as they are.  Only if a norm is off does a second
// pass divide the rows and write the 16-bit ones again.  Bound by memory
// (rows read once, written once and a half).  A block takes 32 rows in slabs
// of 128 columns, a warp four rows of a slab; one warp then adds up the
// squares, a thread per row, from the slab in shared memory, while the others
// load the next slab into the other half.  Device to device: 2,000 x 768 rows
// 26 us, 20,000 x 384 48, 1,000,000 x 768 2,100 (copy, norms, division and
// 16-bit rows as a pass each, with 128 rows to a block: 191, 161 and 5,800).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "batch.h"
#include "common.cuh"
#include "kernels.h"

namespace evoc {

// One f32 value as the 16-bit operand of the tensor-core scan.  FP16: round
// to nearest even, with values below the smallest normal (2^-14) flushed to
// zero, so no subnormal ever reaches the tensor cores and the residual
// x - half(x) below accounts for the whole difference whatever the hardware
// does with subnormal inputs.  BF16: round to nearest even.
__device__ __forceinline__ uint16_t half_bits(float v, int half_type) {
  if (half_type == kHalfBf16) return __bfloat16_as_ushort(__float2bfloat16_rn(v));
  if (fabsf(v) < 6.103515625e-05f) return 0;
  return __half_as_ushort(__float2half_rn(v));
}

__device__ __forceinline__ float half_value(uint16_t b, int half_type) {
  return half_type == kHalfBf16 ? __bfloat162float(__ushort_as_bfloat16(b)) : __half2float(__ushort_as_half(b));
}

namespace {
constexpr int kTileRows = 32;
constexpr int kTileCols = 128;
constexpr int kPrepWarps = 8;
constexpr int kWarpRows = kTileRows / kPrepWarps;
}  // namespace

// One value's share of the two norms the BF16/FP16 form certifies its rows
// with: |x - half(x)| (the residual, exact in f32) and |half(x)|, summed in f64.
__device__ __forceinline__ uint16_t half_and_norms(float v, int half_type, double& rr, double& hh) {
  const uint16_t b = half_bits(v, half_type);
  const float h = half_value(b, half_type);
  const double res = double(__fsub_rn(v, h));  // exact
  rr += res * res;
  hh += double(h) * double(h);
  return b;
}

// A row's sums over its warp, rounded up to f32; their maxima over all rows
// (non-negative floats compare as their bit patterns).
__device__ __forceinline__ void write_cert_norms(double rr, double hh, int lane, float* rnorm, float* hnorm,
                                                 unsigned int* maxes) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    rr += __shfl_xor_sync(0xffffffffu, rr, o);
    hh += __shfl_xor_sync(0xffffffffu, hh, o);
  }
  if (lane == 0) {
    // f64 sums of at most 2^16 squares are within a relative 2^-36 of
    // exact: one part in 2^-30 more before rounding up covers them.
    const float a = __double2float_ru(__dsqrt_ru(rr * (1.0 + 0x1p-30)));
    const float b = __double2float_ru(__dsqrt_ru(hh * (1.0 + 0x1p-30)));
    *rnorm = a;
    *hnorm = b;
    // one address for all rows: only those that raise the maximum take the atomic
    volatile unsigned int* seen = maxes;
    if (__float_as_uint(a) > seen[0]) atomicMax(&maxes[0], __float_as_uint(a));
    if (__float_as_uint(b) > seen[1]) atomicMax(&maxes[1], __float_as_uint(b));
  }
}

// Rows r0 .. r0+31 of one matrix, as they are.
__device__ __forceinline__ void prepare_tile(const PrepRows& p, int64_t r0, float (*slab)[kTileRows][kTileCols + 1]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row0 = r0 + warp * kWarpRows;
  const int64_t width = p.half ? max(p.ld, p.ldb) : p.ld;
  double rr[kWarpRows] = {}, hh[kWarpRows] = {};
  float acc = 0.0f;
  int s = 0;
  for (int64_t c0 = 0; c0 < width; c0 += kTileCols, s ^= 1) {
    float v[kWarpRows][kTileCols / 32];
#pragma unroll
    for (int a = 0; a < kWarpRows; a++)
#pragma unroll
      for (int b = 0; b < kTileCols / 32; b++) {
        const int64_t c = c0 + 32 * b + lane;
        v[a][b] = row0 + a < p.n && c < p.d ? p.src[(row0 + a) * p.src_ld + c] : 0.0f;
      }
#pragma unroll
    for (int a = 0; a < kWarpRows; a++)
#pragma unroll
      for (int b = 0; b < kTileCols / 32; b++) {
        const int64_t r = row0 + a, c = c0 + 32 * b + lane;
        slab[s][warp * kWarpRows + a][32 * b + lane] = v[a][b];
        if (p.src != p.x && c < p.ld) p.x[r * p.ld + c] = v[a][b];
        if (p.half && c < p.ldb) p.half[r * p.ldb + c] = half_and_norms(v[a][b], p.half_type, rr[a], hh[a]);
      }
    __syncthreads();  // this slab is full, and the sums over the one before it are done
    if (warp == 0) {
      const int lim = int(min(int64_t(kTileCols), p.d - c0));
#pragma unroll 8
      for (int c = 0; c < lim; c++) {
        const float x = slab[s][lane][c];
        acc = __fadd_rn(acc, __fmul_rn(x, x));
      }
    }
  }
  if (warp == 0) {
    const bool real = r0 + lane < p.n;
    const float nrm = __fsqrt_rn(acc);
    if (real) p.norms[r0 + lane] = nrm;
    if (__any_sync(0xffffffffu, real && fabsf(__fsub_rn(nrm, 1.0f)) > 1e-5f) && lane == 0) atomicOr(p.not_unit, 1);
  }
  if (p.rnorm) {
#pragma unroll
    for (int a = 0; a < kWarpRows; a++)
      if (row0 + a < p.n) write_cert_norms(rr[a], hh[a], lane, p.rnorm + row0 + a, p.hnorm + row0 + a, p.maxes);
  }
}

// A warp per row: the row divided by its norm, and its 16-bit row again.  The
// maxima gather beside those of the undivided rows, and the last block of
// the grid puts them in their place.
__device__ __forceinline__ void renormalize_rows(const PrepRows& p) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t r = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); r < p.n; r += warps) {
    float nrm = p.norms[r];
    if (nrm == 0.0f) nrm = 1.0f;
    double rr = 0.0, hh = 0.0;
    for (int64_t c = lane; c < p.d; c += 32) {
      const float v = __fdiv_rn(p.x[r * p.ld + c], nrm);
      p.x[r * p.ld + c] = v;
      if (p.half) p.half[r * p.ldb + c] = half_and_norms(v, p.half_type, rr, hh);
    }
    if (p.rnorm) write_cert_norms(rr, hh, lane, p.rnorm + r, p.hnorm + r, p.maxes + 2);
  }
  if (!p.rnorm) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&p.maxes[4], 1u) == gridDim.x - 1) {
    p.maxes[0] = atomicMax(&p.maxes[2], 0u);
    p.maxes[1] = atomicMax(&p.maxes[3], 0u);
  }
}

__global__ void __launch_bounds__(kPrepWarps * 32) prepare_rows_kernel(PrepRows p) {
  __shared__ float slab[2][kTileRows][kTileCols + 1];
  for (int64_t r0 = int64_t(blockIdx.x) * kTileRows; r0 < p.rows; r0 += int64_t(gridDim.x) * kTileRows) {
    prepare_tile(p, r0, slab);
    __syncthreads();
  }
}

__global__ void renormalize_rows_kernel(PrepRows p) {
  if (*p.not_unit != 0) renormalize_rows(p);
}

cudaError_t launch_prepare_rows(const PrepRows& p, int sms, cudaStream_t stream) {
  if (p.rows % kTileRows != 0 || p.rows < p.n || p.src_ld < p.d || p.ld < p.d || (p.half && p.ldb < p.d) ||
      (reinterpret_cast<uintptr_t>(p.src) & 3))
    return cudaErrorInvalidValue;
  if (p.rnorm) {
    cudaError_t e = cudaMemsetAsync(p.maxes, 0, kPrepMaxes * sizeof(unsigned int), stream);
    if (e != cudaSuccess) return e;
  }
  prepare_rows_kernel<<<unsigned(std::min<int64_t>(p.rows / kTileRows, int64_t(sms) * 6)), kPrepWarps * 32, 0,
                        stream>>>(p);
  renormalize_rows_kernel<<<sms * 8, 256, 0, stream>>>(p);
  return cudaGetLastError();
}

// Rows list[i] (+ row0) of src -> row i of dst (row_bytes each, 16-byte
// multiples); dst rows count .. rows_out-1 are zeroed.
__global__ void gather_rows_list_kernel(const uint8_t* __restrict__ src, int64_t row_bytes, int64_t row0,
                                        const int32_t* __restrict__ list, int64_t count, int64_t rows_out,
                                        uint8_t* __restrict__ dst) {
  const int64_t wpr = row_bytes / 16, total = rows_out * wpr;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e / wpr, w = e % wpr;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (i < count) v = reinterpret_cast<const uint4*>(src + (row0 + list[i]) * row_bytes)[w];
    reinterpret_cast<uint4*>(dst + i * row_bytes)[w] = v;
  }
}

cudaError_t launch_gather_rows_list(const void* src, int64_t row_bytes, int64_t row0, const int32_t* list,
                                    int64_t count, int64_t rows_out, void* dst, int sms, cudaStream_t stream) {
  if (row_bytes % 16 != 0 || rows_out < count) return cudaErrorInvalidValue;
  gather_rows_list_kernel<<<sms * 4, 256, 0, stream>>>(static_cast<const uint8_t*>(src), row_bytes, row0, list, count,
                                                       rows_out, static_cast<uint8_t*>(dst));
  return cudaGetLastError();
}

}  // namespace evoc

namespace evoc {

// Row copy with padding.  Wide path: 16-byte words when both strides and
// both base addresses allow it; otherwise 4-byte words; otherwise bytes.
template <typename W>
__global__ void copy_rows_kernel(const uint8_t* __restrict__ src, int64_t n, int64_t row_bytes,
                                 uint8_t* __restrict__ dst, int64_t rows, int64_t ld_bytes) {
  const int64_t wpr = ld_bytes / int64_t(sizeof(W));      // words per destination row
  const int64_t src_w = row_bytes / int64_t(sizeof(W));   // words of data per row
  const int64_t total = rows * wpr;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t r = e / wpr, c = e % wpr;
    W v{};
    if (r < n && c < src_w) v = reinterpret_cast<const W*>(src + r * row_bytes)[c];
    reinterpret_cast<W*>(dst + r * ld_bytes)[c] = v;
  }
}

cudaError_t launch_copy_rows(const void* src, int64_t n, int64_t row_bytes, void* dst, int64_t rows, int64_t ld_bytes,
                             int sms, cudaStream_t stream) {
  if (ld_bytes < row_bytes || rows < n) return cudaErrorInvalidValue;
  const uintptr_t a = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst);
  const auto* s8 = static_cast<const uint8_t*>(src);
  auto* d8 = static_cast<uint8_t*>(dst);
  const int grid = sms * 8;
  if (row_bytes % 16 == 0 && ld_bytes % 16 == 0 && (a & 15) == 0)
    copy_rows_kernel<uint4><<<grid, 256, 0, stream>>>(s8, n, row_bytes, d8, rows, ld_bytes);
  else if (row_bytes % 4 == 0 && ld_bytes % 4 == 0 && (a & 3) == 0)
    copy_rows_kernel<uint32_t><<<grid, 256, 0, stream>>>(s8, n, row_bytes, d8, rows, ld_bytes);
  else
    copy_rows_kernel<uint8_t><<<grid, 256, 0, stream>>>(s8, n, row_bytes, d8, rows, ld_bytes);
  return cudaGetLastError();
}

}  // namespace evoc

// ---------------------------------------------------------------------------
// Batches: the same per-request steps over the request table of a batch.
// ---------------------------------------------------------------------------
namespace evoc {

namespace {
__device__ __forceinline__ int find_block_job(const BatchRowJob* __restrict__ jobs, int nj, int64_t g) {
  int lo = 0, hi = nj - 1;
  while (lo < hi) {  // last request with blk_base <= g
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].blk_base <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
}  // namespace

// Packed int8 rows -> padded rows (xb, ldb bytes), zero-filled past the data.
__global__ void batch_copy_kernel(const BatchHeader* __restrict__ hdr, const BatchRowJob* __restrict__ jobs) {
  const int nj = hdr->n_jobs;
  for (int j = 0; j < nj; j++) {
    const BatchRowJob& J = jobs[j];
    if (J.row_bytes % 4 == 0) {
      const int64_t wpr = J.ldb / 4, src_w = J.row_bytes / 4, total = J.rows * wpr;
      for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
           e += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = e / wpr, c = e % wpr;
        uint32_t v = 0u;
        if (r < J.n && c < src_w) v = reinterpret_cast<const uint32_t*>(J.src + r * J.row_bytes)[c];
        reinterpret_cast<uint32_t*>(J.xb + r * J.ldb)[c] = v;
      }
    } else {
      const int64_t total = J.rows * J.ldb;
      for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
           e += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = e / J.ldb, c = e % J.ldb;
        J.xb[e] = (r < J.n && c < J.row_bytes) ? J.src[r * J.row_bytes + c] : uint8_t(0);
      }
    }
  }
}

__device__ __forceinline__ PrepRows job_rows(const BatchRowJob& J) {
  PrepRows p{};
  p.src = reinterpret_cast<const float*>(J.src);
  p.src_ld = J.row_bytes / 4;
  p.x = J.x;
  p.n = J.n;
  p.rows = J.rows;
  p.d = J.dim;
  p.ld = J.ld;
  p.norms = J.norms;
  p.not_unit = J.flag;
  p.half = reinterpret_cast<uint16_t*>(J.xb);
  p.ldb = J.ldb / 2;
  p.half_type = J.half_type;
  p.rnorm = J.rnorm;
  p.hnorm = J.hnorm;
  p.maxes = J.maxes;
  return p;
}

__global__ void batch_clear_kernel(const BatchHeader* __restrict__ hdr, const BatchRowJob* __restrict__ jobs) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < hdr->n_jobs; j += gridDim.x * blockDim.x) {
    *jobs[j].flag = 0;
    if (jobs[j].maxes)
      for (int i = 0; i < kPrepMaxes; i++) jobs[j].maxes[i] = 0u;
  }
}

__global__ void __launch_bounds__(kPrepWarps * 32)
batch_prepare_kernel(const BatchHeader* __restrict__ hdr, const BatchRowJob* __restrict__ jobs) {
  __shared__ float slab[2][kTileRows][kTileCols + 1];
  const int nj = hdr->n_jobs;
  const int64_t total = hdr->total_blocks;
  for (int64_t g = blockIdx.x; g < total; g += gridDim.x) {
    const BatchRowJob& J = jobs[find_block_job(jobs, nj, g)];
    prepare_tile(job_rows(J), (g - J.blk_base) * kTileRows, slab);
    __syncthreads();
  }
}

__global__ void batch_renormalize_kernel(const BatchHeader* __restrict__ hdr, const BatchRowJob* __restrict__ jobs) {
  const int nj = hdr->n_jobs;
  for (int j = 0; j < nj; j++)
    if (*jobs[j].flag != 0) renormalize_rows(job_rows(jobs[j]));
}

cudaError_t launch_batch_rows(bool f32, const BatchHeader* hdr, const BatchRowJob* jobs, int grid_rows,
                              int grid_tiles, cudaStream_t stream) {
  if (!f32) {
    batch_copy_kernel<<<grid_rows, 256, 0, stream>>>(hdr, jobs);
    return cudaGetLastError();
  }
  batch_clear_kernel<<<1, 256, 0, stream>>>(hdr, jobs);
  batch_prepare_kernel<<<grid_tiles, kPrepWarps * 32, 0, stream>>>(hdr, jobs);
  batch_renormalize_kernel<<<grid_rows, 256, 0, stream>>>(hdr, jobs);
  return cudaGetLastError();
}

}  // namespace evoc

namespace evoc {

namespace {
__device__ __forceinline__ uint64_t fill_hash(uint64_t z) {  // splitmix64 finaliser
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
}  // namespace

__global__ void fill_random_kernel(int mode, uint8_t* __restrict__ rows, int64_t n_rows_mem, int64_t row_bytes,
                                   int64_t n, int64_t bytes, uint64_t seed) {
  const int64_t total = n_rows_mem * row_bytes;
  const int64_t eb = mode == 0 ? 2 : 1;
  for (int64_t e = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * eb; e < total;
       e += int64_t(gridDim.x) * blockDim.x * eb) {
    const int64_t r = e / row_bytes, c = e % row_bytes;
    const bool live = r < n && c < bytes;
    const uint64_t h = fill_hash(seed ^ uint64_t(e));
    if (mode == 0) {
      const float v = live ? float(int32_t(h & 0xffff) - 32768) / 32768.0f : 0.0f;
      *reinterpret_cast<__half*>(rows + e) = __float2half_rn(v);
    } else if (mode == 1) {
      rows[e] = live ? uint8_t(int8_t(int32_t(h % 255) - 127)) : uint8_t(0);
    } else {
      const uint64_t b = h & (h >> 8) & (h >> 16);  // each bit set with probability 1/8
      rows[e] = live ? uint8_t(b) : uint8_t(0);
    }
  }
}

cudaError_t launch_fill_random(int mode, void* rows, int64_t n_rows_mem, int64_t row_bytes, int64_t n,
                               int64_t bytes, uint64_t seed, int sms, cudaStream_t stream) {
  if (mode < 0 || mode > 2 || (mode == 0 && (row_bytes % 2 || bytes % 2))) return cudaErrorInvalidValue;
  fill_random_kernel<<<sms * 8, 256, 0, stream>>>(mode, static_cast<uint8_t*>(rows), n_rows_mem, row_bytes, n, bytes,
                                                  seed);
  return cudaGetLastError();
}

}  // namespace evoc
