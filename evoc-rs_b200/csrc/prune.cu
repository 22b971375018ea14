// Tile lists for the exact self-join: which 256-row key tiles a query block
// has to multiply, and which provably hold none of its rows' neighbours.
//
// The rows are scanned in an order that puts like rows side by side: every
// row goes to its nearest pivot (n/512 evenly spaced rows), and the pivots are
// visited as Prim's algorithm adds them to a maximum spanning tree of their
// similarities, so whatever clusters the data has at whatever scale lie in
// one run each.  Rows far less similar to their pivot than the closer rows of
// its cell (those above the cell's mean) are strays, members of clusters too small to have drawn a pivot;
// one stray opens its whole tile, so the strays get pivots of their own
// (every 64th) in a second round.  A group is `g` consecutive tiles (g = 1 up
// to 2^20 rows).  Where the order passes from one cluster to the next inside
// a group (a pivot is added at a similarity under 0.75 of its cell's own), the
// group is cut there: a segment is what lies between two cuts or group ends,
// with a centre m, the mean of its rows rounded to the operand type.
//
// Bound.  With x = a_x m_A + x' for a row x of segment A (a_x = x.m_A / |m_A|^2,
// x' orthogonal to m_A), for q in A and k in B
//   q.k = a_q (k.m_A) + a_k (q.m_B - a_q m_A.m_B) + q'.k'
// and q'.k' <= |q'| |k'|.  Per segment the smallest and largest a and the
// largest |x'| are known, per pair of segments the largest x.m_B over x in A
// (one product of the rows with the centres, the column maxima taken in its
// epilogue) and m_A.m_B.  A pair is skipped when the bound stays below the
// smallest of its query rows' thresholds; groups multiply when any pair of
// their segments does.  A row's threshold is a score that keep other rows among
// the 512 around the row's block reach (seed_kernel).  A skipped key
// then scores strictly below keep keys of the row, so the kept sets are those
// of the full scan, ties included.
//
// Where rows are not alike enough for the bound to skip anything, or no more
// unlike the others than they are alike (a sample's cosines with the pivots
// tell), the full scan runs instead.
//
// Slack.  The products with the centres and the scores the bound is compared
// with are tensor-core sums: at most e = (L/4 + 2) 2^-21 |x||y| off for 16-bit
// operands of length L, exact for integers.  The bound adds up five such
// terms of size at most N^2 (N the largest row norm).  The a_x are off by the
// f32 sums that make them, (L/32 + L/512 + 28) 2^-24 of |x| / |m|, and stand in
// three terms.  16-bit rows get 16 e N^2, of which 11 e cover the latter;
// integer rows 8 (L/32 + L/512) 2^-24 N^2 (their sums are exact up to about
// 1,040 features); both 1e-5 N^2 for the operations on the sums.  The |x'|
// carry an allowance of their own (segment_stats_kernel).  For binary rows the
// bound on the intersection becomes one on J through the segments' smallest
// popcounts.
//
// Replaces nothing in the reference, which prunes by its RP forest and
// NN-descent (src/nndescent/float.rs:775-879) without a guarantee.
#include <algorithm>
#include <cfloat>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "batch.h"
#include "common.cuh"
#include "kernels.h"
#include "sm100.cuh"

namespace evoc {

namespace {
constexpr int BM = 128;  // rows per block
constexpr int BN = 256;  // centres per tile
constexpr int KCB = 128;
constexpr int A_BYTES = BM * KCB;
constexpr int STAGE_BYTES = A_BYTES + BN * KCB;
constexpr int STAGES = 4;
constexpr size_t kSmem = size_t(STAGES) * STAGE_BYTES + 1024 + 256;

struct ProductParams {
  int64_t rows, n_ctiles;  // rows of A; tiles of 256 centres
  int n_kchunks, half_type;
  Segments seg;            // column maxima are per segment
  void* out;               // kStore: f32 [rows][ld]; else int32 [segments][ld], maxima with 0
  int64_t ld;
  int* status;
  uint64_t timeout_ns, drain_ns;
};
}  // namespace

// Rows x centres on the tensor cores (the scan's pipeline: TMA producer warp,
// MMA warp, four epilogue warps, two accumulators).  kStore writes the
// products (kBits: as the accumulator holds them, s32 for int8); otherwise
// each column's maximum over a segment's rows, as the
// signed pattern of a non-negative f32 or s32.  At 1M x 768 against 3,907
// centres: 6 TFLOP.
template <bool kInt8, bool kStore, bool kBits = false>
__global__ void __launch_bounds__(192, 1)
centre_product_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const ProductParams p) {
  using namespace sm100;
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = smem_dyn + ((1024u - (smem_addr(smem_dyn) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* mma_done = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 128);
    }
    mbar_init(mma_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int64_t items = (p.rows + BM - 1) / BM * p.n_ctiles;
  const volatile int* abort = p.status;
  constexpr int KC_ELEMS = kInt8 ? KCB : KCB / 2;
  const uint32_t idesc = kInt8 ? idesc_s8_s32(BM, BN)
                               : (p.half_type == kHalfBf16 ? idesc_bf16_f32(BM, BN) : idesc_f16_f32(BM, BN));
  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int64_t i = blockIdx.x; ok && i < items; i += gridDim.x) {
        const int32_t row = int32_t(i / p.n_ctiles * BM), centre = int32_t(i % p.n_ctiles * BN);
        for (int kc = 0; kc < p.n_kchunks; kc++, it++) {
          const uint32_t s = it % STAGES;
          if (!mbar_wait(&empty[s], ((it / STAGES) & 1u) ^ 1u, abort, p.timeout_ns)) {
            atomicCAS(p.status, 0, 1);
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
          tma_load_2d(smem + s * STAGE_BYTES, &tmA, &full[s], kc * KC_ELEMS, row);
          tma_load_2d(smem + s * STAGE_BYTES + A_BYTES, &tmB, &full[s], kc * KC_ELEMS, centre);
        }
      }
      // the last loads land before the CTA can exit
      for (uint32_t j = (it > STAGES ? it - STAGES : 0); j < it; j++)
        mbar_wait(&full[j % STAGES], (j / STAGES) & 1u, nullptr, p.drain_ns);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t it = 0, tile = 0;
      bool ok = true;
      for (int64_t i = blockIdx.x; ok && i < items; i += gridDim.x, tile++) {
        const uint32_t a = tile & 1u;
        if (!mbar_wait(&tempty[a], ((tile >> 1) & 1u) ^ 1u, abort, p.timeout_ns)) {
          atomicCAS(p.status, 0, 2);
          break;
        }
        tc_fence_after();
        for (int kc = 0; kc < p.n_kchunks; kc++, it++) {
          const uint32_t s = it % STAGES;
          if (!mbar_wait(&full[s], (it / STAGES) & 1u, abort, p.timeout_ns)) {
            atomicCAS(p.status, 0, 2);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_addr(smem + s * STAGE_BYTES);
          const uint64_t ad = sw128_kmajor_desc(sa), bd = sw128_kmajor_desc(sa + A_BYTES);
#pragma unroll
          for (int j = 0; j < KCB / 32; j++) {
            const uint32_t acc = (kc > 0 || j > 0) ? 1u : 0u;
            if (kInt8) mma_i8(tmem_base + a * BN, ad + 2 * j, bd + 2 * j, idesc, acc);
            else mma_f16(tmem_base + a * BN, ad + 2 * j, bd + 2 * j, idesc, acc);
          }
          mma_commit(&empty[s]);
        }
        if (!ok) break;
        mma_commit(&tfull[a]);
      }
      mma_commit(mma_done);
      mbar_wait(mma_done, 0, nullptr, p.drain_ns);
    }
  } else {
    const int quad = warp & 3;
    uint32_t tile = 0;
    int64_t last = -1;
    int32_t seg = 0;
    for (int64_t i = blockIdx.x; i < items; i += gridDim.x, tile++) {
      const uint32_t a = tile & 1u;
      if (!kStore && i / p.n_ctiles != last) {  // the lane's row's segment
        last = i / p.n_ctiles;
        const int64_t r = min(last * BM + quad * 32 + lane, p.rows - 1);  // rows past the data are zero
        seg = p.seg.first[r / p.seg.group_rows];
        while (p.seg.start[seg + 1] <= r) seg++;
      }
      int got = 1;
      if (lane == 0) got = mbar_wait(&tfull[a], (tile >> 1) & 1u, abort, p.timeout_ns) ? 1 : 0;
      if (!__shfl_sync(0xffffffffu, got, 0)) {
        if (lane == 0) atomicCAS(p.status, 0, 3);
        break;
      }
      tc_fence_after();
      const int64_t row = i / p.n_ctiles * BM + quad * 32 + lane, col0 = i % p.n_ctiles * BN;
      const uint32_t taddr = tmem_base + (uint32_t(quad * 32) << 16) + a * BN;
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(taddr + c, v);
        tmem_ld_wait();
        if (kStore) {
          if (row < p.rows) {
            float4* o = reinterpret_cast<float4*>(static_cast<float*>(p.out) + row * p.ld + col0 + c);
#pragma unroll
            for (int j = 0; j < 8; j++) {
              float f[4];
#pragma unroll
              for (int u = 0; u < 4; u++)
                f[u] = kInt8 && !kBits ? __int2float_rn(int32_t(v[4 * j + u])) : __uint_as_float(v[4 * j + u]);
              o[j] = make_float4(f[0], f[1], f[2], f[3]);
            }
          }
        } else {
          // the warp's rows mostly share a segment: one round
          uint32_t todo = 0xffffffffu;
          while (todo) {
            const int32_t sg = __shfl_sync(0xffffffffu, seg, __ffs(todo) - 1);
            todo &= ~__ballot_sync(0xffffffffu, seg == sg);
            int32_t mine = 0;  // lane j: column j's maximum
#pragma unroll
            for (int j = 0; j < 32; j++) {
              const int32_t m = __reduce_max_sync(0xffffffffu, seg == sg ? int32_t(v[j]) : 0);
              if (lane == j) mine = m;
            }
            if (mine > 0) atomicMax(static_cast<int32_t*>(p.out) + int64_t(sg) * p.ld + col0 + c + lane, mine);
          }
        }
      }
      tc_fence_before();
      mbar_arrive(&tempty[a]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// A seed for every row: a score that at least `keep` other rows among the 512
// around its block (192 before, 192 after) reach.  Their scores stay in TMEM
// (512 columns) and every lane bisects for its row by counting over them, 13
// passes; scanning as many keys with key sets spends ten times as long, most
// of it on the first keys.  One block of 128 rows at a time per CTA.
constexpr int kBefore = 192;

struct SeedParams {
  int64_t n;
  int n_kchunks, half_type, keep;
  float eps;                // 16-bit scores: twice the products' error relative to the largest |x|^2
  const unsigned int* top;  // the largest |x|^2 (f32 bits)
  const int32_t* pc;        // popcounts (Jaccard)
  float* seed;              // per row, a dissimilarity (kHeapInf: none)
  int* status;
  uint64_t timeout_ns, drain_ns;
};

// mode 0: 16-bit dots, 1: int8 dots, 2: Jaccard of 0/1 rows.
template <int MODE>
__global__ void __launch_bounds__(192, 1)
seed_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const SeedParams p) {
  using namespace sm100;
  constexpr bool kInt8 = MODE != kScanHalf;
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = smem_dyn + ((1024u - (smem_addr(smem_dyn) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 1;
  uint64_t* mma_done = tempty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
  __shared__ float sizes[MODE == kScanJaccard ? 2 * BN : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, 128);
    mbar_init(mma_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int64_t blocks = (p.n + BM - 1) / BM;
  const volatile int* abort = p.status;
  constexpr int KC_ELEMS = kInt8 ? KCB : KCB / 2;
  const uint32_t idesc = kInt8 ? idesc_s8_s32(BM, BN)
                               : (p.half_type == kHalfBf16 ? idesc_bf16_f32(BM, BN) : idesc_f16_f32(BM, BN));
  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int64_t qb = blockIdx.x; ok && qb < blocks; qb += gridDim.x)
        for (int i = 0; ok && i < 2; i++) {
          const int32_t row = int32_t(qb * BM), key = row - kBefore + i * BN;  // rows outside the data read as zero
          for (int kc = 0; kc < p.n_kchunks; kc++, it++) {
            const uint32_t s = it % STAGES;
            if (!mbar_wait(&empty[s], ((it / STAGES) & 1u) ^ 1u, abort, p.timeout_ns)) {
              atomicCAS(p.status, 0, 1);
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
            tma_load_2d(smem + s * STAGE_BYTES, &tmA, &full[s], kc * KC_ELEMS, row);
            tma_load_2d(smem + s * STAGE_BYTES + A_BYTES, &tmB, &full[s], kc * KC_ELEMS, key);
          }
        }
      for (uint32_t j = (it > STAGES ? it - STAGES : 0); j < it; j++)
        mbar_wait(&full[j % STAGES], (j / STAGES) & 1u, nullptr, p.drain_ns);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t it = 0, done = 0;
      bool ok = true;
      for (int64_t qb = blockIdx.x; ok && qb < blocks; qb += gridDim.x, done++) {
        if (!mbar_wait(tempty, (done & 1u) ^ 1u, abort, p.timeout_ns)) {
          atomicCAS(p.status, 0, 2);
          break;
        }
        tc_fence_after();
        for (int i = 0; ok && i < 2; i++)
          for (int kc = 0; kc < p.n_kchunks; kc++, it++) {
            const uint32_t s = it % STAGES;
            if (!mbar_wait(&full[s], (it / STAGES) & 1u, abort, p.timeout_ns)) {
              atomicCAS(p.status, 0, 2);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_addr(smem + s * STAGE_BYTES);
            const uint64_t ad = sw128_kmajor_desc(sa), bd = sw128_kmajor_desc(sa + A_BYTES);
#pragma unroll
            for (int j = 0; j < KCB / 32; j++) {
              const uint32_t acc = (kc > 0 || j > 0) ? 1u : 0u;
              if (kInt8) mma_i8(tmem_base + i * BN, ad + 2 * j, bd + 2 * j, idesc, acc);
              else mma_f16(tmem_base + i * BN, ad + 2 * j, bd + 2 * j, idesc, acc);
            }
            mma_commit(&empty[s]);
          }
        if (!ok) break;
        mma_commit(tfull);
      }
      mma_commit(mma_done);
      mbar_wait(mma_done, 0, nullptr, p.drain_ns);
    }
  } else {
    const int quad = warp & 3;
    uint32_t done = 0;
    for (int64_t qb = blockIdx.x; qb < blocks; qb += gridDim.x, done++) {
      int got = 1;
      if (lane == 0) got = mbar_wait(tfull, done & 1u, abort, p.timeout_ns) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got && lane == 0) atomicCAS(p.status, 0, 3);
      // the four warps stop together: they share the barrier below
      uint32_t all;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 128, q;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}\n"
          : "=r"(all)
          : "r"(uint32_t(got))
          : "memory");
      if (!all) break;
      tc_fence_after();
      if (MODE == kScanJaccard) {
        for (int c = quad * 32 + lane; c < 2 * BN; c += 128) {
          const int64_t key = qb * BM - kBefore + c;
          sizes[c] = key >= 0 && key < p.n ? float(p.pc[key]) : 0.0f;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
      const int64_t row = qb * BM + quad * 32 + lane;
      const uint32_t taddr = tmem_base + (uint32_t(quad * 32) << 16);
      const float pa = MODE == kScanJaccard && row < p.n ? float(p.pc[row]) : 0.0f;
      // Scores of the row above t (J above t: inter above t / (1 + t) times the
      // two sizes); zero rows past the data never are, t being non-negative.
      auto count = [&](float t, float* most) {
        int c = 0;
        float mx = 0.0f;
        const float share = t / (1.0f + t), own = share * pa;
#pragma unroll 1
        for (int a = 0; a < 2 * BN; a += 32) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(taddr + a, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j++) {
            const float s = kInt8 ? __int2float_rn(int32_t(v[j])) : __uint_as_float(v[j]);
            c += s > (MODE == kScanJaccard ? fmaf(share, sizes[a + j], own) : t) ? 1 : 0;
            if (most) mx = fmaxf(mx, s);
          }
        }
        if (most) *most = mx;
        return c;
      };
      float hi = 0.0f;
      const int positive = count(0.0f, &hi);  // the row itself among them
      if (MODE == kScanJaccard) hi = 1.0f;
      float lo = 0.0f;
      const bool some = positive > p.keep;
#pragma unroll 1
      for (int i = 0; i < 12; i++) {
        const float mid = 0.5f * (lo + hi);
        if (count(mid, nullptr) > p.keep) lo = mid;
        else hi = mid;
      }
      if (MODE == kScanHalf) lo -= p.eps * __uint_as_float(*p.top);
      else lo *= 1.0f - 1e-5f;
      if (row < p.n) p.seed[row] = some && lo > 0.0f ? -lo : kHeapInf;
      tc_fence_before();
      mbar_arrive(tempty);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

namespace {

// Visits the pivots as Prim's algorithm does, each time the one most similar
// to any visited so far: a cluster of pivots at any similarity is one run.
// One block, four pivots a thread; a step is one row of the similarities
// (shared memory where the matrix fits it, else L2) and one block maximum.
// Similarity and pivot share a word (20 and 12 bits: the order need not be
// exact), so a maximum is one reduction a warp and one more over the warps,
// with a single barrier between (two sets of warp results alternate).
// Bound by that chain: ~0.35 us a step from shared memory, ~0.6 from L2.
constexpr int kPrimThreads = 1024;
constexpr int kPrimMax = 4096;
constexpr int kPrimShared = 224;  // largest matrix kept in shared memory

template <bool kShared>
__global__ void __launch_bounds__(kPrimThreads)
prim_order_kernel(const float* __restrict__ sim, int64_t ld, int n, int active, int32_t* __restrict__ rank,
                  float* __restrict__ attach) {
  extern __shared__ float matrix[];
  __shared__ uint32_t part[2][32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, warps = active >> 5;
  if (kShared) {  // all threads load, `active` of them go on
    for (int r = warp; r < n; r += int(blockDim.x) >> 5)
#pragma unroll 4
      for (int c = lane; c < n; c += 32) matrix[r * n + c] = sim[int64_t(r) * ld + c];
    __syncthreads();
    if (t >= active) return;
  }
  uint32_t best[4];  // orderable similarity to the visited ones; 0: visited or past the end
#pragma unroll
  for (int u = 0; u < 4; u++) best[u] = t + u * active < n ? 1u << 12 : 0u;
  int cur = 0;
  float with = 0.0f;  // the similarity the current pivot was added at
  for (int step = 0; step < n; step++) {
    if (t == 0) {
      rank[cur] = step;
      attach[step] = with;
    }
    const float* row = kShared ? matrix + cur * n : sim + int64_t(cur) * ld;
    float v[4];  // all loads before the first use
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = row[min(t + u * active, n - 1)];
    uint32_t top = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int j = t + u * active;
      if (best[u] != 0u) best[u] = j == cur ? 0u : max(best[u], orderable(v[u]));
      if (best[u] != 0u) top = max(top, (best[u] & ~0xfffu) | uint32_t(kPrimMax - 1 - j));
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (warps > 1) {
      if (lane == 0) part[step & 1][warp] = top;
      asm volatile("bar.sync 1, %0;" ::"r"(active) : "memory");
      top = __reduce_max_sync(0xffffffffu, lane < warps ? part[step & 1][lane] : 0u);
    }
    if (top == 0u) break;  // all visited
    cur = kPrimMax - 1 - int(top & 0xfffu);
    with = from_orderable(top & ~0xfffu);
  }
}

// A warp's sum of squares of an int8 row (row_bytes a multiple of 16).
__device__ __forceinline__ int row_sq(const uint8_t* row, int64_t row_bytes, int lane) {
  const int4* x = reinterpret_cast<const int4*>(row);
  int s = 0;
  for (int c = lane; c < row_bytes / 16; c += 32) {
    const int4 v = x[c];
    s = __dp4a(v.x, v.x, s);
    s = __dp4a(v.y, v.y, s);
    s = __dp4a(v.z, v.z, s);
    s = __dp4a(v.w, v.w, s);
  }
  return __reduce_add_sync(0xffffffffu, s);
}

// Squared norms of int8 rows, warp per row.
__global__ void int8_sq_kernel(const uint8_t* __restrict__ rows, int64_t row_bytes, int64_t n, int32_t* __restrict__ sq) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t r = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps) {
    const int s = row_sq(rows + r * row_bytes, row_bytes, lane);
    if (lane == 0) sq[r] = s;
  }
}

// Cosine of row i with its pivot.  Pivot p is row floor(p n / n_piv); map
// (optional) leads from both to the rows sq is about.
__device__ __forceinline__ float pivot_cosine(int64_t i, int32_t label, int n_piv, int64_t n, const float* raw,
                                              const int32_t* sq, const int32_t* map) {
  const float s = fmaxf(-raw[i], 0.0f);
  if (!sq) return s;  // unit rows
  const int64_t p = int64_t(label) * n / n_piv;
  const float w = float(sq[map ? map[i] : i]) * float(sq[map ? map[p] : p]);
  return w > 0.0f ? s * rsqrtf(w) : 0.0f;
}

// Squared norms of the sampled rows, then of the sampled pivots (int8 rows), warp per row.
__global__ void sample_sq_kernel(const uint8_t* __restrict__ rows, int64_t row_bytes, Sample s,
                                 int32_t* __restrict__ sq) {
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < s.rows + s.pivots; i += warps) {
    const int64_t r = i < s.rows ? s.first + i * s.stride : (i - s.rows) * s.pivot_stride;
    const int v = row_sq(rows + r * row_bytes, row_bytes, lane);
    if (lane == 0) sq[i] = v;
  }
}

// Counts the sampled rows that the lists may serve, warp per row: with c the
// cosine with the nearest pivot and b the mean over all pivots (0 at least),
// those with 1 - c below `part` of 1 - b.
__global__ void sample_fit_kernel(const float* __restrict__ products, int64_t ld, Sample s,
                                  const int32_t* __restrict__ sq, float part, int32_t* __restrict__ fit) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= s.rows) return;
  const float* row = products + i * ld;
  const float own = sq ? rsqrtf(fmaxf(float(sq[i]), 1.0f)) : 1.0f;  // f32 rows have unit length
  const int64_t self = s.first + i * s.stride;
  float most = 0.0f, sum = 0.0f;
  for (int p = lane; p < s.pivots; p += 32) {
    if (p * s.pivot_stride == self) continue;  // the row itself is a pivot
    const float c = row[p] * own * (sq ? rsqrtf(fmaxf(float(sq[s.rows + p]), 1.0f)) : 1.0f);
    most = fmaxf(most, c);
    sum += c;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if (lane == 0 && 1.0f - most < part * (1.0f - fmaxf(sum / float(s.pivots), 0.0f))) atomicAdd(fit, 1);
}

// Per cell the sum of its rows' cosines with the pivot and their number; with
// all_sum / all_count (an earlier call's), of the rows above the cell's mean.
__global__ void cell_fit_kernel(const int32_t* __restrict__ label, const float* __restrict__ raw, int64_t n, int n_piv,
                                const int32_t* __restrict__ sq, const int32_t* __restrict__ map,
                                const float* __restrict__ all_sum, const int32_t* __restrict__ all_count,
                                float* __restrict__ sum, int32_t* __restrict__ count) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t b = min(max(label[i], 0), n_piv - 1);
    const float c = pivot_cosine(i, b, n_piv, n, raw, sq, map);
    if (all_sum && c < all_sum[b] / float(max(all_count[b], 1))) continue;
    atomicAdd(&sum[b], c);
    atomicAdd(&count[b], 1);
  }
}

// Rows whose cosine is under 0.6 of the given mean; the other rows' sums.
__global__ void strays_kernel(const int32_t* __restrict__ label, const float* __restrict__ raw, int64_t n, int n_piv,
                              const int32_t* __restrict__ sq, const float* __restrict__ sum,
                              const int32_t* __restrict__ count, float* __restrict__ own_sum,
                              int32_t* __restrict__ own_count, int32_t* __restrict__ list,
                              int32_t* __restrict__ strays) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t b = min(max(label[i], 0), n_piv - 1);
    const float c = pivot_cosine(i, b, n_piv, n, raw, sq, nullptr);
    if (c < 0.6f * sum[b] / float(max(count[b], 1))) {
      list[atomicAdd(strays, 1)] = int32_t(i);
    } else {
      atomicAdd(&own_sum[b], c);
      atomicAdd(&own_count[b], 1);
    }
  }
}

__global__ void stray_labels_kernel(const int32_t* __restrict__ list, const int32_t* __restrict__ second, int64_t count,
                                    int first, int n_second, int32_t* __restrict__ label) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += int64_t(gridDim.x) * blockDim.x)
    label[list[i]] = first + min(max(second[i], 0), n_second - 1);
}

__global__ void relabel_kernel(int32_t* __restrict__ label, int64_t n, const int32_t* __restrict__ rank, int nb) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t b = label[i];
    label[i] = rank[b < 0 || b >= nb ? 0 : b];
  }
}

// The segments: group starts and, merged in, the starts of cells that begin a
// cluster.  One block.  cell c (in rank order) holds rows [end[c] - size[c],
// end[c]); room: segments the arrays hold.
__global__ void __launch_bounds__(1024)
segments_kernel(const int32_t* __restrict__ rank, const float* __restrict__ attach, const float* __restrict__ own_sum,
                const int32_t* __restrict__ own_count, int n_piv, const int32_t* __restrict__ end,
                const int32_t* __restrict__ size, int64_t n, int64_t group_rows, int groups, int room,
                int32_t* __restrict__ cuts, Segments seg, int32_t* __restrict__ n_seg, int32_t* __restrict__ group_of) {
  __shared__ uint8_t begins[kPrimMax];
  __shared__ int32_t part[1024];
  const int t = threadIdx.x;
  for (int c = t; c < n_piv; c += 1024) {
    const int r = rank[c];
    const float own = own_sum[c] / float(max(own_count[c], 1));
    begins[r] = r > 0 && own_count[c] > 0 && attach[r] < 0.75f * own ? 1 : 0;
  }
  __syncthreads();
  const int per = (n_piv + 1023) / 1024;
  int mine = 0;
  for (int i = 0; i < per; i++) {
    const int c = t * per + i;
    if (c >= n_piv) break;
    const int64_t at = int64_t(end[c]) - size[c];
    if (size[c] == 0 || at <= 0 || at >= n || at % group_rows == 0) begins[c] = 0;
    mine += begins[c];
  }
  part[t] = mine;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const int32_t v = t >= off ? part[t - off] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  const int n_cuts = min(part[1023], room - groups);
  int at = part[t] - mine;
  for (int i = 0; i < per; i++) {
    const int c = t * per + i;
    if (c >= n_piv) break;
    if (begins[c]) {
      if (at < n_cuts) cuts[at] = end[c] - size[c];  // cells are in row order, so the cuts ascend
      at++;
    }
  }
  __syncthreads();
  // merge: a group start's place is its index plus the cuts before it, and the other way round
  for (int g = t; g <= groups; g += 1024) {
    const int64_t s = g < groups ? int64_t(g) * group_rows : n;
    int lo = 0, hi = n_cuts;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (cuts[mid] < s) lo = mid + 1;
      else hi = mid;
    }
    seg.start[g + lo] = int32_t(s);
    if (g < groups) {
      seg.first[g] = g + lo;
      group_of[g + lo] = g;
    } else {
      seg.first[groups] = g + lo;
      *n_seg = groups + n_cuts;
    }
  }
  for (int i = t; i < n_cuts; i += 1024) {
    const int g = int(cuts[i] / group_rows);  // its group's start lies before it
    seg.start[i + g + 1] = cuts[i];
    group_of[i + g + 1] = g;
  }
}

// The 16 bytes at word w of a row: 8 16-bit or 16 int8 values.
template <bool kInt8>
struct Lane16 {
  static constexpr int N = kInt8 ? 16 : 8;
  float v[N];
  __device__ __forceinline__ Lane16(const uint8_t* row, int w, int half_type) {
    const uint4 q = reinterpret_cast<const uint4*>(row)[w];
    const uint32_t r[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < N; i++) {
      if (kInt8) {
        v[i] = float(int8_t(r[i >> 2] >> (8 * (i & 3))));
      } else {
        const uint16_t h = uint16_t(r[i >> 1] >> (16 * (i & 1)));
        v[i] = half_type == kHalfBf16 ? __bfloat162float(__ushort_as_bfloat16(h)) : __half2float(__ushort_as_half(h));
      }
    }
  }
};

// One block per segment: its centre (16-bit: the mean scaled to unit length;
// int8: scaled to a largest entry of 127), then per row a_x and |x'|.
// Two passes over the segment's rows, the second from L2.
constexpr int kStatThreads = 512;

template <bool kInt8>
__global__ void __launch_bounds__(kStatThreads)
segment_stats_kernel(const uint8_t* __restrict__ rows, int64_t row_bytes, Segments seg, int half_type,
                     uint8_t* __restrict__ centres, PruneStats st) {
  extern __shared__ float mean[];  // one value per element of a row, then the centre's values
  __shared__ float red[kStatThreads / 32][4];
  const int len = int(kInt8 ? row_bytes : row_bytes / 2);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t A = blockIdx.x, r0 = seg.start[A], r1 = seg.start[A + 1];
  using Vec = Lane16<kInt8>;
  for (int c = t; c < len; c += kStatThreads) mean[c] = 0.0f;
  __syncthreads();
  for (int w = lane; w < row_bytes / 16; w += 32) {  // each warp its rows, 16 bytes of a row a lane
    float s[Vec::N];
#pragma unroll
    for (int i = 0; i < Vec::N; i++) s[i] = 0.0f;
#pragma unroll 4
    for (int64_t r = r0 + warp; r < r1; r += kStatThreads / 32) {
      const Vec x(rows + r * row_bytes, w, half_type);
#pragma unroll
      for (int i = 0; i < Vec::N; i++) s[i] += x.v[i];
    }
#pragma unroll
    for (int i = 0; i < Vec::N; i++) atomicAdd(&mean[w * Vec::N + i], s[i]);
  }
  __syncthreads();
  float acc_max = 0.0f, acc_sq = 0.0f;
  for (int c = t; c < len; c += kStatThreads) {
    acc_max = fmaxf(acc_max, fabsf(mean[c]));
    acc_sq += mean[c] * mean[c];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc_max = fmaxf(acc_max, __shfl_xor_sync(0xffffffffu, acc_max, o));
    acc_sq += __shfl_xor_sync(0xffffffffu, acc_sq, o);
  }
  if (lane == 0) {
    red[warp][0] = acc_max;
    red[warp][1] = acc_sq;
  }
  __syncthreads();
  acc_max = acc_sq = 0.0f;
  for (int w = 0; w < kStatThreads / 32; w++) {
    acc_max = fmaxf(acc_max, red[w][0]);
    acc_sq += red[w][1];
  }
  __syncthreads();
  const float scale = kInt8 ? (acc_max > 0.0f ? 127.0f / acc_max : 0.0f) : (acc_sq > 0.0f ? rsqrtf(acc_sq) : 0.0f);
  float msq = 0.0f;
  for (int c = t; c < len; c += kStatThreads) {
    float v = mean[c] * scale;
    if (kInt8) {
      v = rintf(v);
      reinterpret_cast<int8_t*>(centres + A * row_bytes)[c] = int8_t(v);
    } else {
      uint16_t b;
      if (half_type == kHalfBf16) b = __bfloat16_as_ushort(__float2bfloat16_rn(v));
      else b = fabsf(v) < 6.103515625e-05f ? uint16_t(0) : __half_as_ushort(__float2half_rn(v));  // no subnormals
      reinterpret_cast<uint16_t*>(centres + A * row_bytes)[c] = b;
      v = half_type == kHalfBf16 ? __bfloat162float(__ushort_as_bfloat16(b)) : __half2float(__ushort_as_half(b));
    }
    mean[c] = v;
    msq += v * v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) msq += __shfl_xor_sync(0xffffffffu, msq, o);
  if (lane == 0) red[warp][0] = msq;
  __syncthreads();
  msq = 0.0f;
  for (int w = 0; w < kStatThreads / 32; w++) msq += red[w][0];
  __syncthreads();
  // |x'|^2 = sq - dot^2 / msq cancels, so the sums' rounding counts against |x|^2: sq is off by
  // (L/32 + 5) u of it (a lane's chain and five additions), dot^2 by twice that, msq by (L/512 + 23) u;
  // the last operations take 9 u more.
  const float allowance = (3.0f * float((len + 31) / 32) + float(len) / 512.0f + 48.0f) * 0x1p-24f;
  float a0 = FLT_MAX, a1 = -FLT_MAX, rho = 0.0f, nsq = 0.0f, sq0 = FLT_MAX;
  for (int64_t r = r0 + warp; r < r1; r += kStatThreads / 32) {
    const uint8_t* row = rows + r * row_bytes;
    float dot = 0.0f, sq = 0.0f;
#pragma unroll 2
    for (int w = lane; w < row_bytes / 16; w += 32) {
      const Vec x(row, w, half_type);
#pragma unroll
      for (int i = 0; i < Vec::N; i++) {
        dot = fmaf(x.v[i], mean[w * Vec::N + i], dot);
        sq = fmaf(x.v[i], x.v[i], sq);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dot += __shfl_xor_sync(0xffffffffu, dot, o);
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
    }
    const float a = msq > 0.0f ? dot / msq : 0.0f;
    a0 = fminf(a0, a);
    a1 = fmaxf(a1, a);
    rho = fmaxf(rho, sqrtf(fmaxf(sq - a * dot, 0.0f) + allowance * sq));
    nsq = fmaxf(nsq, sq);
    sq0 = fminf(sq0, sq);
  }
  if (lane == 0) {
    red[warp][0] = a0;
    red[warp][1] = a1;
    red[warp][2] = rho;
    red[warp][3] = nsq;
  }
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < kStatThreads / 32; w++) {
      a0 = fminf(a0, red[w][0]);
      a1 = fmaxf(a1, red[w][1]);
      rho = fmaxf(rho, red[w][2]);
      nsq = fmaxf(nsq, red[w][3]);
    }
    st.a0[A] = a0;
    st.a1[A] = a1;
    st.rho[A] = rho;
  }
  __syncthreads();
  if (lane == 0) red[warp][0] = sq0;
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < kStatThreads / 32; w++) sq0 = fminf(sq0, red[w][0]);
    st.sq0[A] = sq0;
    atomicMax(st.top, __float_as_uint(nsq));  // non-negative floats order as their bits
  }
}

// One block per group: the ascending list of groups it has to multiply.
constexpr int kDecideThreads = 256;

__global__ void __launch_bounds__(kDecideThreads)
decide_kernel(int mode, Segments seg, const int32_t* __restrict__ group_of, int segments, int groups, int64_t ld,
              const int32_t* __restrict__ U, const float* __restrict__ G, PruneStats st, const float* __restrict__ T,
              int half_len, int32_t* __restrict__ list, int32_t* __restrict__ len) {
  __shared__ float red[kDecideThreads / 32];
  __shared__ int base, counts[kDecideThreads / 32];
  __shared__ uint32_t hit[kPruneGroups / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = blockIdx.x;
  for (int i = t; i < kPruneGroups / 32; i += kDecideThreads) hit[i] = 0u;
  const float nn = __uint_as_float(*st.top);
  // 16-bit: 16 e; integers, whose products are exact: eight times what their f32 sums are off by
  const float e = mode == kScanHalf ? (float(half_len) / 4.0f + 2.0f) * 0x1p-21f * 16.0f
                                    : 8.0f * (float(half_len) / 16.0f + float(half_len) / 256.0f) * 0x1p-24f;
  const float slack = (e + 1e-5f) * nn;
  auto value = [&](int32_t u) { return mode == kScanHalf ? __int_as_float(u) : float(u); };
  __syncthreads();
  for (int A = seg.first[g]; A < seg.first[g + 1]; A++) {
    // the smallest of the rows' thresholds, as a score (-FLT_MAX: no bound)
    float thr = FLT_MAX;
    for (int r = seg.start[A] + t; r < seg.start[A + 1]; r += kDecideThreads) {
      const float raw = T[r];
      const bool none = raw == kHeapInf || (mode != kScanInt8 && raw >= 0.0f);
      thr = fminf(thr, none ? -FLT_MAX : -raw);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) thr = fminf(thr, __shfl_xor_sync(0xffffffffu, thr, o));
    __syncthreads();
    if (lane == 0) red[warp] = thr;
    __syncthreads();
    for (int w = 0; w < kDecideThreads / 32; w++) thr = fminf(thr, red[w]);
    const float a0 = st.a0[A], a1 = st.a1[A], rho = st.rho[A], sqa = st.sq0[A];
    for (int B = t; B < segments; B += kDecideThreads) {
      const float uab = value(U[A * ld + B]), uba = value(U[B * ld + A]), gab = G[A * ld + B];
      const float c0 = st.a0[B], c1 = st.a1[B];
      const float w = uab - fminf(a0 * gab, a1 * gab);
      const float top = a1 * uba + fmaxf(c0 * w, c1 * w) + rho * st.rho[B] + slack;
      // a row turned against its centre leaves the bound's sign cases: keep the pair
      bool in = A == B || a0 < 0.0f || c0 < 0.0f || !(thr > -FLT_MAX);
      if (!in && mode == kScanJaccard) {
        const float size = sqa + st.sq0[B] - top;  // J <= i / (|a| + |b| - i), increasing in i
        in = !(size > 0.0f) || top >= thr * size * (1.0f - 1e-5f);
      } else if (!in) {
        in = !(top < thr);
      }
      if (in) {
        const int h = group_of[B];
        if (!(hit[h >> 5] >> (h & 31) & 1u)) atomicOr(&hit[h >> 5], 1u << (h & 31));
      }
    }
  }
  if (t == 0) base = 0;
  __syncthreads();
  for (int b0 = 0; b0 < groups; b0 += kDecideThreads) {
    const int b = b0 + t;
    const bool in = b < groups && (hit[b >> 5] >> (b & 31) & 1u);
    const uint32_t who = __ballot_sync(0xffffffffu, in);
    if (lane == 0) counts[warp] = __popc(who);
    __syncthreads();
    int at = base;
    for (int w = 0; w < warp; w++) at += counts[w];
    if (in) list[int64_t(g) * groups + at + __popc(who & ((1u << lane) - 1u))] = b;
    __syncthreads();
    if (t == 0)
      for (int w = 0; w < kDecideThreads / 32; w++) base += counts[w];
    __syncthreads();
  }
  if (t == 0) len[g] = base;
}

// The query blocks by descending list length (counting sort in one block):
// dealt in turns forth and back, every CTA then gets about the same work.
// *total: the tiles of all blocks.
__global__ void __launch_bounds__(1024)
block_order_kernel(const int32_t* __restrict__ len, int groups, int64_t n_blocks, int blocks_per_group,
                   int32_t* __restrict__ order, unsigned long long* __restrict__ total) {
  extern __shared__ int32_t bins[];  // groups + 1, longest first
  __shared__ int32_t part[1024];
  const int t = threadIdx.x, nb = groups + 1;
  for (int b = t; b < nb; b += blockDim.x) bins[b] = 0;
  __syncthreads();
  unsigned long long tiles = 0;
  for (int64_t q = t; q < n_blocks; q += blockDim.x) {
    const int32_t l = len[q / blocks_per_group];
    atomicAdd(&bins[groups - l], 1);
    tiles += (unsigned long long)(l) * unsigned(blocks_per_group / 2);  // a tile: two blocks of rows
  }
  atomicAdd(total, tiles);
  __syncthreads();
  const int per = (nb + blockDim.x - 1) / blockDim.x;
  int32_t s = 0;
  for (int i = 0; i < per; i++)
    if (t * per + i < nb) s += bins[t * per + i];
  part[t] = s;
  __syncthreads();
  for (int off = 1; off < int(blockDim.x); off <<= 1) {
    const int32_t v = t >= off ? part[t - off] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  int32_t run = part[t] - s;
  for (int i = 0; i < per; i++)
    if (t * per + i < nb) {
      const int32_t c = bins[t * per + i];
      bins[t * per + i] = run;
      run += c;
    }
  __syncthreads();
  for (int64_t q = t; q < n_blocks; q += blockDim.x)
    order[atomicAdd(&bins[groups - len[q / blocks_per_group]], 1)] = int32_t(q);
}

}  // namespace

cudaError_t launch_centre_products(int mode, const void* A, int64_t a_rows_mem, int64_t rows, const void* C,
                                   int64_t c_rows_mem, int64_t row_bytes, int half_type, const Segments* seg,
                                   void* out, int64_t ld, int* status, uint64_t timeout_ns, int sms,
                                   cudaStream_t stream, bool bits) {
  if (row_bytes % KCB || rows < 1 || a_rows_mem < rows || c_rows_mem % BN || ld < c_rows_mem || ld % 4)
    return cudaErrorInvalidValue;
  const bool store = seg == nullptr;
  const int eb = mode == kScanHalf ? 2 : 1;
  alignas(64) CUtensorMap ma, mb;
  if (!encode_row_map(&ma, A, a_rows_mem, row_bytes, eb, BM, half_type) ||
      !encode_row_map(&mb, C, c_rows_mem, row_bytes, eb, BN, half_type))
    return cudaErrorInvalidValue;
  ProductParams p{};
  p.rows = rows;
  p.n_ctiles = c_rows_mem / BN;
  p.n_kchunks = int(row_bytes / KCB);
  p.half_type = half_type;
  if (seg) p.seg = *seg;
  p.out = out;
  p.ld = ld;
  p.status = status;
  p.timeout_ns = timeout_ns;
  p.drain_ns = timeout_ns > 4000000000ull ? timeout_ns : 4000000000ull;
  const int64_t items = (rows + BM - 1) / BM * p.n_ctiles;
  const unsigned grid = unsigned(items < sms ? items : sms);
  auto go = [&](auto kern) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
    if (e != cudaSuccess) return e;
    kern<<<grid, 192, kSmem, stream>>>(ma, mb, p);
    return cudaGetLastError();
  };
  if (mode == kScanHalf) return store ? go(centre_product_kernel<false, true>) : go(centre_product_kernel<false, false>);
  if (store && bits) return go(centre_product_kernel<true, true, true>);
  return store ? go(centre_product_kernel<true, true>) : go(centre_product_kernel<true, false>);
}

cudaError_t launch_seeds(int mode, const void* X, int64_t rows_mem, int64_t n, int64_t row_bytes, int keep,
                         int half_type, const unsigned int* top, const int32_t* pc, float* seed, int* status,
                         uint64_t timeout_ns, int grid, cudaStream_t stream) {
  if (row_bytes % KCB || n < 1 || rows_mem < n || rows_mem % BN || (mode == kScanJaccard && !pc))
    return cudaErrorInvalidValue;
  const int eb = mode == kScanHalf ? 2 : 1;
  alignas(64) CUtensorMap ma, mb;
  if (!encode_row_map(&ma, X, rows_mem, row_bytes, eb, BM, half_type) ||
      !encode_row_map(&mb, X, rows_mem, row_bytes, eb, BN, half_type))
    return cudaErrorInvalidValue;
  SeedParams p{};
  p.n = n;
  p.n_kchunks = int(row_bytes / KCB);
  p.half_type = half_type;
  p.keep = keep;
  p.eps = 2.0f * (float(row_bytes / 2) / 4.0f + 2.0f) * 0x1p-21f;
  p.top = top;
  p.pc = pc;
  p.seed = seed;
  p.status = status;
  p.timeout_ns = timeout_ns;
  p.drain_ns = timeout_ns > 4000000000ull ? timeout_ns : 4000000000ull;
  auto go = [&](auto kern) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
    if (e != cudaSuccess) return e;
    kern<<<unsigned(grid), 192, kSmem, stream>>>(ma, mb, p);
    return cudaGetLastError();
  };
  if (mode == kScanHalf) return go(seed_kernel<kScanHalf>);
  return mode == kScanInt8 ? go(seed_kernel<kScanInt8>) : go(seed_kernel<kScanJaccard>);
}

cudaError_t launch_int8_sq(const void* rows, int64_t row_bytes, int64_t n, int32_t* sq, int sms, cudaStream_t stream) {
  if (row_bytes % 16) return cudaErrorInvalidValue;
  int8_sq_kernel<<<sms * 8, 256, 0, stream>>>(static_cast<const uint8_t*>(rows), row_bytes, n, sq);
  return cudaGetLastError();
}

Sample list_sample(int64_t n, int64_t n_piv) {
  Sample s{};
  s.rows = 1024;
  s.stride = n / s.rows;
  s.first = s.stride / 2;
  s.pivots = int(n_piv);
  s.pivot_stride = n / n_piv;
  return s;
}

size_t sample_fit_bytes(const Sample& s) {
  return size_t(s.rows) * size_t((s.pivots + BN - 1) / BN * BN) * 4 + size_t(s.rows + s.pivots) * 4 + 256;
}

cudaError_t launch_sample_fit(int mode, const void* rows, int64_t row_bytes, int half_type, const Sample& s, float part,
                              void* work, int32_t** fit, int* status, uint64_t timeout_ns, int sms,
                              cudaStream_t stream) {
  if (row_bytes % KCB || s.rows % BM || s.stride < 1 || s.pivot_stride < 1) return cudaErrorInvalidValue;
  const bool half = mode == kScanHalf;
  const int eb = half ? 2 : 1;
  alignas(64) CUtensorMap ma, mb;
  if (!encode_row_map(&ma, static_cast<const uint8_t*>(rows) + s.first * row_bytes, s.rows, row_bytes, eb, BM, half_type,
                      s.stride * row_bytes) ||
      !encode_row_map(&mb, rows, s.pivots, row_bytes, eb, BN, half_type, s.pivot_stride * row_bytes))
    return cudaErrorInvalidValue;
  ProductParams p{};
  p.rows = s.rows;
  p.n_ctiles = (s.pivots + BN - 1) / BN;
  p.n_kchunks = int(row_bytes / KCB);
  p.half_type = half_type;
  p.ld = p.n_ctiles * BN;
  int32_t* counter = static_cast<int32_t*>(work);
  float* products = reinterpret_cast<float*>(counter + 64);
  int32_t* sq = half ? nullptr : reinterpret_cast<int32_t*>(products + s.rows * p.ld);
  p.out = products;
  p.status = status;
  p.timeout_ns = timeout_ns;
  p.drain_ns = timeout_ns > 4000000000ull ? timeout_ns : 4000000000ull;
  cudaError_t e = cudaMemsetAsync(counter, 0, 4, stream);
  if (e != cudaSuccess) return e;
  if (sq) sample_sq_kernel<<<sms * 2, 256, 0, stream>>>(static_cast<const uint8_t*>(rows), row_bytes, s, sq);
  const int64_t items = s.rows / BM * p.n_ctiles;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
    if (e != cudaSuccess) return e;
    kern<<<unsigned(std::min<int64_t>(items, sms)), 192, kSmem, stream>>>(ma, mb, p);
    return cudaGetLastError();
  };
  e = half ? go(centre_product_kernel<false, true>) : go(centre_product_kernel<true, true>);
  if (e != cudaSuccess) return e;
  sample_fit_kernel<<<(s.rows + 7) / 8, 256, 0, stream>>>(products, p.ld, s, sq, part, counter);
  *fit = counter;
  return cudaGetLastError();
}

cudaError_t launch_cell_fit(const int32_t* label, const float* raw, int64_t n, int n_piv, const int32_t* sq,
                            const int32_t* map, const float* all_sum, const int32_t* all_count, float* sum,
                            int32_t* count, int sms, cudaStream_t stream) {
  cell_fit_kernel<<<sms * 4, 256, 0, stream>>>(label, raw, n, n_piv, sq, map, all_sum, all_count, sum, count);
  return cudaGetLastError();
}

cudaError_t launch_strays(const int32_t* label, const float* raw, int64_t n, int n_piv, const int32_t* sq,
                          const float* sum, const int32_t* count, float* own_sum, int32_t* own_count, int32_t* list,
                          int32_t* strays, int sms, cudaStream_t stream) {
  strays_kernel<<<sms * 4, 256, 0, stream>>>(label, raw, n, n_piv, sq, sum, count, own_sum, own_count, list, strays);
  return cudaGetLastError();
}

cudaError_t launch_segments(const int32_t* rank, const float* attach, const float* own_sum, const int32_t* own_count,
                            int n_piv, const int32_t* end, const int32_t* size, int64_t n, int64_t group_rows,
                            int groups, int room, int32_t* cuts, const Segments& seg, int32_t* n_seg,
                            int32_t* group_of, cudaStream_t stream) {
  if (n_piv < 1 || n_piv > kPrimMax || room < groups) return cudaErrorInvalidValue;
  segments_kernel<<<1, 1024, 0, stream>>>(rank, attach, own_sum, own_count, n_piv, end, size, n, group_rows, groups,
                                          room, cuts, seg, n_seg, group_of);
  return cudaGetLastError();
}

cudaError_t launch_stray_labels(const int32_t* list, const int32_t* second, int64_t count, int first, int n_second,
                                int32_t* label, int sms, cudaStream_t stream) {
  stray_labels_kernel<<<sms * 2, 256, 0, stream>>>(list, second, count, first, n_second, label);
  return cudaGetLastError();
}

cudaError_t launch_prim_order(const float* sim, int64_t ld, int n, int32_t* rank, float* attach, int32_t* label,
                              int64_t n_rows, int sms, cudaStream_t stream) {
  if (n < 1 || n > kPrimMax) return cudaErrorInvalidValue;
  const int threads = ((n + 3) / 4 + 31) / 32 * 32;
  if (n <= kPrimShared) {
    const cudaError_t e = cudaFuncSetAttribute(prim_order_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kPrimShared * kPrimShared * 4);
    if (e != cudaSuccess) return e;
    prim_order_kernel<true><<<1, kPrimThreads, size_t(n) * n * 4, stream>>>(sim, ld, n, threads, rank, attach);
  } else {
    prim_order_kernel<false><<<1, threads, 0, stream>>>(sim, ld, n, threads, rank, attach);
  }
  relabel_kernel<<<sms * 4, 256, 0, stream>>>(label, n_rows, rank, n);
  return cudaGetLastError();
}

cudaError_t launch_segment_stats(int mode, const void* rows, int64_t row_bytes, const Segments& seg, int segments,
                                 int half_type, void* centres, const PruneStats& st, cudaStream_t stream) {
  const int len = int(mode == kScanHalf ? row_bytes / 2 : row_bytes);
  const size_t smem = size_t(len) * sizeof(float);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(st.top, 0, 4, stream);
  if (e != cudaSuccess) return e;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    kern<<<unsigned(segments), kStatThreads, smem, stream>>>(static_cast<const uint8_t*>(rows), row_bytes, seg,
                                                             half_type, static_cast<uint8_t*>(centres), st);
    return cudaGetLastError();
  };
  return mode == kScanHalf ? go(segment_stats_kernel<false>) : go(segment_stats_kernel<true>);
}

cudaError_t launch_prune_lists(int mode, int64_t n, int64_t group_rows, int groups, const Segments& seg,
                               const int32_t* group_of, int segments, int64_t ld, const int32_t* U, const float* G,
                               const PruneStats& st, const float* T, int half_len, int32_t* list, int32_t* len,
                               int32_t* block_order, unsigned long long* tiles, cudaStream_t stream) {
  if (groups < 1 || groups > kPruneGroups || segments < groups) return cudaErrorInvalidValue;
  decide_kernel<<<unsigned(groups), kDecideThreads, 0, stream>>>(mode, seg, group_of, segments, groups, ld, U, G, st,
                                                                 T, half_len, list, len);
  block_order_kernel<<<1, 1024, size_t(groups + 1) * 4, stream>>>(len, groups, (n + BM - 1) / BM,
                                                                  int(group_rows / BM), block_order, tiles);
  return cudaGetLastError();
}

}  // namespace evoc
