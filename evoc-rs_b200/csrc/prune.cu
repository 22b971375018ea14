// Tile lists for the exact self-join: which 256-row key tiles a query block
// has to multiply, and which provably hold none of its rows' neighbours.
//
// The rows are scanned in an order that puts like rows side by side: every
// row goes to its nearest pivot (n/512 evenly spaced rows), and the pivots are
// visited as Prim's algorithm adds them to a maximum spanning tree of their
// similarities, so whatever clusters the data has at whatever scale lie in
// one run each.  Rows far less similar to their pivot than the other rows of
// its cell are strays, members of clusters too small to have drawn a pivot;
// one stray opens its whole tile, so the strays get pivots of their own
// (every 64th) in a second round.  A group is `g` consecutive tiles (g = 1 up
// to 2^20 rows) with a centre m, the mean of its rows rounded to the operand
// type.
//
// Bound.  With x = a_x m_A + x' for a row x of group A (a_x = x.m_A / |m_A|^2,
// x' orthogonal to m_A), for q in A and k in B
//   q.k = a_q (k.m_A) + a_k (q.m_B - a_q m_A.m_B) + q'.k'
// and q'.k' <= |q'| |k'|.  Per group the smallest and largest a and the
// largest |x'| are known, per pair of groups the largest x.m_B over x in A
// (one product of the rows with the centres, the column maxima taken in its
// epilogue) and m_A.m_B.  A pair is skipped when the bound stays below the
// smallest of its query rows' thresholds: a score that keep other rows among
// the 512 around the row's block reach (seed_kernel).  A skipped key
// then scores strictly below keep keys of the row, so the kept sets are those
// of the full scan, ties included.
//
// Where rows are not alike enough for the bound to skip anything (a sample's
// cosines with the pivots tell), the full scan runs instead.
//
// Slack.  The products with the centres and the scores the bound is compared
// with are tensor-core sums: at most e = (L/4 + 2) 2^-21 |x||y| off for 16-bit
// operands of length L, exact for integers.  The bound adds up five such
// terms of size at most N^2 (N the largest row norm); it is given 16 e N^2 and
// 1e-5 N^2 more for the f32 arithmetic here.  For binary rows the bound on
// the intersection becomes one on J through the groups' smallest popcounts.
//
// Replaces nothing in the reference, which prunes by its RP forest and
// NN-descent (src/nndescent/float.rs:775-879) without a guarantee.
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
  int64_t group_rows;      // rows per group (column maxima)
  void* out;               // kStore: f32 [rows][ld]; else int32 [groups][ld], maxima with 0
  int64_t ld;
  int* status;
  uint64_t timeout_ns, drain_ns;
};
}  // namespace

// Rows x centres on the tensor cores (the scan's pipeline: TMA producer warp,
// MMA warp, four epilogue warps, two accumulators).  kStore writes the
// products; otherwise each column's maximum over the group's rows, as the
// signed pattern of a non-negative f32 or s32.  At 1M x 768 against 3,907
// centres: 6 TFLOP.
template <bool kInt8, bool kStore>
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
    for (int64_t i = blockIdx.x; i < items; i += gridDim.x, tile++) {
      const uint32_t a = tile & 1u;
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
                f[u] = kInt8 ? __int2float_rn(int32_t(v[4 * j + u])) : __uint_as_float(v[4 * j + u]);
              o[j] = make_float4(f[0], f[1], f[2], f[3]);
            }
          }
        } else {
          int32_t mine = 0;  // lane j: column j's maximum (rows past the data are zero)
#pragma unroll
          for (int j = 0; j < 32; j++) {
            const int32_t m = __reduce_max_sync(0xffffffffu, int32_t(v[j]));
            if (lane == j) mine = m;
          }
          if (mine > 0)
            atomicMax(static_cast<int32_t*>(p.out) + i / p.n_ctiles * BM / p.group_rows * p.ld + col0 + c + lane,
                      mine);
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
// One block; a step is one row of the similarities (from L2) and a block
// maximum with a single barrier (two sets of warp results alternate).
constexpr int kPrimThreads = 1024;
constexpr int kPrimMax = 4096;

__global__ void __launch_bounds__(kPrimThreads)
prim_order_kernel(const float* __restrict__ sim, int64_t ld, int n, int32_t* __restrict__ rank) {
  __shared__ unsigned long long part[2][kPrimThreads / 32];
  constexpr int PER = kPrimMax / kPrimThreads;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t best[PER];  // orderable similarity to the visited ones; 0: visited or past the end
#pragma unroll
  for (int u = 0; u < PER; u++) best[u] = t + u * kPrimThreads < n ? 1u : 0u;
  int cur = 0;
  for (int step = 0; step < n; step++) {
    if (t == 0) rank[cur] = step;
    uint32_t top = 0;
    int at = 0;
    float v[PER];  // all loads before the first use: a step is one L2 round trip
#pragma unroll
    for (int u = 0; u < PER; u++) v[u] = sim[int64_t(cur) * ld + min(t + u * kPrimThreads, n - 1)];
#pragma unroll
    for (int u = 0; u < PER; u++) {
      const int j = t + u * kPrimThreads;
      if (best[u] != 0u) best[u] = j == cur ? 0u : max(best[u], max(orderable(v[u]), 1u));
      if (best[u] > top) {
        top = best[u];
        at = j;
      }
    }
    const uint32_t wtop = __reduce_max_sync(0xffffffffu, top);
    const uint32_t wat = __reduce_min_sync(0xffffffffu, top == wtop ? uint32_t(at) : 0xffffffffu);
    if (lane == 0) part[step & 1][warp] = (static_cast<unsigned long long>(wtop) << 32) | wat;
    __syncthreads();
    const unsigned long long w = part[step & 1][lane];
    const uint32_t btop = __reduce_max_sync(0xffffffffu, uint32_t(w >> 32));
    cur = int(__reduce_min_sync(0xffffffffu, uint32_t(w >> 32) == btop ? uint32_t(w) : 0xffffffffu));
    if (btop == 0u) break;  // all visited
  }
}

// Squared norms of int8 rows (row_bytes a multiple of 16), warp per row.
__global__ void int8_sq_kernel(const uint8_t* __restrict__ rows, int64_t row_bytes, int64_t n, int32_t* __restrict__ sq) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t r = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps) {
    const int4* x = reinterpret_cast<const int4*>(rows + r * row_bytes);
    int s = 0;
    for (int c = lane; c < row_bytes / 16; c += 32) {
      const int4 v = x[c];
      s = __dp4a(v.x, v.x, s);
      s = __dp4a(v.y, v.y, s);
      s = __dp4a(v.z, v.z, s);
      s = __dp4a(v.w, v.w, s);
    }
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) sq[r] = s;
  }
}

__device__ __forceinline__ float pivot_cosine(int64_t i, int32_t label, int n_piv, int64_t n, const float* raw,
                                              const int32_t* sq) {
  const float s = fmaxf(-raw[i], 0.0f);
  if (!sq) return s;  // unit rows
  const float w = float(sq[i]) * float(sq[int64_t(label) * n / n_piv]);  // pivot p is row floor(p n / n_piv)
  return w > 0.0f ? s * rsqrtf(w) : 0.0f;
}

// Of m sampled rows (sample i is row i * stride) those whose cosine with their
// pivot reaches `least`.
__global__ void sample_fit_kernel(const int32_t* __restrict__ label, const float* __restrict__ raw, int m,
                                  int64_t stride, int64_t n, int n_piv, const int32_t* __restrict__ sq, float least,
                                  int32_t* __restrict__ close) {
  int c = 0;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const int32_t b = min(max(label[i], 0), n_piv - 1);
    float s = fmaxf(-raw[i], 0.0f);
    if (sq) s *= rsqrtf(fmaxf(float(sq[i * stride]) * float(sq[int64_t(b) * n / n_piv]), 1.0f));
    c += s >= least ? 1 : 0;
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) atomicAdd(close, c);
}

// Per cell the sum of its rows' cosines with the pivot and their number.
__global__ void cell_fit_kernel(const int32_t* __restrict__ label, const float* __restrict__ raw, int64_t n, int n_piv,
                                const int32_t* __restrict__ sq, CellFit f) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t b = min(max(label[i], 0), n_piv - 1);
    atomicAdd(&f.sum[b], pivot_cosine(i, b, n_piv, n, raw, sq));
    atomicAdd(&f.count[b], 1);
  }
}

// Rows whose cosine is under 0.6 of their cell's mean.
__global__ void strays_kernel(const int32_t* __restrict__ label, const float* __restrict__ raw, int64_t n, int n_piv,
                              const int32_t* __restrict__ sq, CellFit f, int32_t* __restrict__ list) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int32_t b = min(max(label[i], 0), n_piv - 1);
    if (pivot_cosine(i, b, n_piv, n, raw, sq) < 0.6f * f.sum[b] / float(max(f.count[b], 1)))
      list[atomicAdd(f.strays, 1)] = int32_t(i);
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

__device__ __forceinline__ float half_at(const uint8_t* row, int c, int half_type) {
  const uint16_t b = reinterpret_cast<const uint16_t*>(row)[c];
  return half_type == kHalfBf16 ? __bfloat162float(__ushort_as_bfloat16(b)) : __half2float(__ushort_as_half(b));
}

template <bool kInt8>
__device__ __forceinline__ float elem(const uint8_t* row, int c, int half_type) {
  return kInt8 ? float(reinterpret_cast<const int8_t*>(row)[c]) : half_at(row, c, half_type);
}

// One block per group: its centre (16-bit: the mean scaled to unit length;
// int8: scaled to a largest entry of 127), then per row a_x and |x'|.
// Two passes over the group's rows, the second from L2.
constexpr int kStatThreads = 256;

template <bool kInt8>
__global__ void __launch_bounds__(kStatThreads)
group_stats_kernel(const uint8_t* __restrict__ rows, int64_t row_bytes, int64_t n, int64_t group_rows, int half_type,
                   uint8_t* __restrict__ centres, PruneStats st) {
  extern __shared__ float mean[];  // one value per element of a row, then the centre's values
  __shared__ float red[kStatThreads / 32][4];
  const int len = int(kInt8 ? row_bytes : row_bytes / 2);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t A = blockIdx.x, r0 = A * group_rows, r1 = min(n, r0 + group_rows);
  float acc_max = 0.0f, acc_sq = 0.0f;
  for (int c = t; c < len; c += kStatThreads) {
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int64_t r = r0;
    for (; r + 4 <= r1; r += 4)
#pragma unroll
      for (int u = 0; u < 4; u++) s[u] += elem<kInt8>(rows + (r + u) * row_bytes, c, half_type);
    for (; r < r1; r++) s[0] += elem<kInt8>(rows + r * row_bytes, c, half_type);
    const float m = (s[0] + s[1]) + (s[2] + s[3]);
    mean[c] = m;
    acc_max = fmaxf(acc_max, fabsf(m));
    acc_sq += m * m;
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
  float a0 = FLT_MAX, a1 = -FLT_MAX, rho = 0.0f, nsq = 0.0f, sq0 = FLT_MAX;
  for (int64_t r = r0 + warp; r < r1; r += kStatThreads / 32) {
    const uint8_t* row = rows + r * row_bytes;
    float dot = 0.0f, sq = 0.0f;
    for (int c = lane; c < len; c += 32) {
      const float x = elem<kInt8>(row, c, half_type);
      dot = fmaf(x, mean[c], dot);
      sq = fmaf(x, x, sq);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dot += __shfl_xor_sync(0xffffffffu, dot, o);
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
    }
    const float a = msq > 0.0f ? dot / msq : 0.0f;
    a0 = fminf(a0, a);
    a1 = fmaxf(a1, a);
    // the subtraction cancels: 4e-6 |x|^2 covers the sums' rounding
    rho = fmaxf(rho, sqrtf(fmaxf(sq - a * dot, 0.0f) + 4e-6f * sq));
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

// One block per group A: the ascending list of groups B it has to multiply.
constexpr int kDecideThreads = 256;

__global__ void __launch_bounds__(kDecideThreads)
decide_kernel(int mode, int64_t n, int64_t group_rows, int groups, int64_t ld, const int32_t* __restrict__ U,
              const float* __restrict__ G, PruneStats st, const float* __restrict__ T, int half_len,
              int32_t* __restrict__ list, int32_t* __restrict__ len) {
  __shared__ float red[kDecideThreads / 32];
  __shared__ int base, counts[kDecideThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, A = blockIdx.x;
  // the smallest of the rows' thresholds, as a score (-FLT_MAX: no bound)
  float thr = FLT_MAX;
  for (int64_t r = A * group_rows + t; r < min(n, (A + 1) * group_rows); r += kDecideThreads) {
    const float raw = T[r];
    const bool none = raw == kHeapInf || (mode != kScanInt8 && raw >= 0.0f);
    thr = fminf(thr, none ? -FLT_MAX : -raw);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) thr = fminf(thr, __shfl_xor_sync(0xffffffffu, thr, o));
  if (lane == 0) red[warp] = thr;
  if (t == 0) base = 0;
  __syncthreads();
  for (int w = 0; w < kDecideThreads / 32; w++) thr = fminf(thr, red[w]);
  const float nn = __uint_as_float(*st.top);
  const float e = mode == kScanHalf ? (float(half_len) / 4.0f + 2.0f) * 0x1p-21f * 16.0f : 0.0f;
  const float slack = (e + 1e-5f) * nn;
  const float a0 = st.a0[A], a1 = st.a1[A], rho = st.rho[A], sqa = st.sq0[A];
  auto value = [&](int32_t u) { return mode == kScanHalf ? __int_as_float(u) : float(u); };
  for (int b0 = 0; b0 < groups; b0 += kDecideThreads) {
    const int B = b0 + t;
    bool in = false;
    if (B < groups) {
      const float uab = value(U[A * ld + B]), uba = value(U[B * ld + A]), g = G[A * ld + B];
      const float c0 = st.a0[B], c1 = st.a1[B];
      const float w = uab - fminf(a0 * g, a1 * g);
      const float top = a1 * uba + fmaxf(c0 * w, c1 * w) + rho * st.rho[B] + slack;
      // a row against its centre (never seen) leaves the bound's sign cases: keep the pair
      in = A == B || a0 < 0.0f || c0 < 0.0f || !(thr > -FLT_MAX);
      if (!in && mode == kScanJaccard) {
        const float size = sqa + st.sq0[B] - top;  // J <= i / (|a| + |b| - i), increasing in i
        in = !(size > 0.0f) || top >= thr * size * (1.0f - 1e-5f);
      } else if (!in) {
        in = !(top < thr);
      }
    }
    const uint32_t who = __ballot_sync(0xffffffffu, in);
    if (lane == 0) counts[warp] = __popc(who);
    __syncthreads();
    int at = base;
    for (int w = 0; w < warp; w++) at += counts[w];
    if (in) list[int64_t(A) * groups + at + __popc(who & ((1u << lane) - 1u))] = B;
    __syncthreads();
    if (t == 0)
      for (int w = 0; w < kDecideThreads / 32; w++) base += counts[w];
    __syncthreads();
  }
  if (t == 0) len[A] = base;
}

// The query blocks by descending list length (counting sort in one block):
// dealt in turns forth and back, every CTA then gets about the same work.
__global__ void __launch_bounds__(1024)
block_order_kernel(const int32_t* __restrict__ len, int groups, int64_t n_blocks, int blocks_per_group,
                   int32_t* __restrict__ order) {
  extern __shared__ int32_t bins[];  // groups + 1, longest first
  __shared__ int32_t part[1024];
  const int t = threadIdx.x, nb = groups + 1;
  for (int b = t; b < nb; b += blockDim.x) bins[b] = 0;
  __syncthreads();
  for (int64_t q = t; q < n_blocks; q += blockDim.x) atomicAdd(&bins[groups - len[q / blocks_per_group]], 1);
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
                                   int64_t c_rows_mem, int64_t row_bytes, int half_type, bool store,
                                   int64_t group_rows, void* out, int64_t ld, int* status, uint64_t timeout_ns,
                                   int sms, cudaStream_t stream) {
  if (row_bytes % KCB || rows < 1 || a_rows_mem < rows || c_rows_mem % BN || ld < c_rows_mem || ld % 4 ||
      group_rows % BM)
    return cudaErrorInvalidValue;
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
  p.group_rows = group_rows;
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

cudaError_t launch_sample_fit(const int32_t* label, const float* raw, int m, int64_t stride, int64_t n, int n_piv,
                              const int32_t* sq, float least, int32_t* close, cudaStream_t stream) {
  if (m < 1 || (m - 1) * stride >= n) return cudaErrorInvalidValue;
  sample_fit_kernel<<<1, 1024, 0, stream>>>(label, raw, m, stride, n, n_piv, sq, least, close);
  return cudaGetLastError();
}

cudaError_t launch_cell_fit(const int32_t* label, const float* raw, int64_t n, int n_piv, const int32_t* sq,
                            const CellFit& f, int32_t* list, int sms, cudaStream_t stream) {
  cell_fit_kernel<<<sms * 4, 256, 0, stream>>>(label, raw, n, n_piv, sq, f);
  strays_kernel<<<sms * 4, 256, 0, stream>>>(label, raw, n, n_piv, sq, f, list);
  return cudaGetLastError();
}

cudaError_t launch_stray_labels(const int32_t* list, const int32_t* second, int64_t count, int first, int n_second,
                                int32_t* label, int sms, cudaStream_t stream) {
  stray_labels_kernel<<<sms * 2, 256, 0, stream>>>(list, second, count, first, n_second, label);
  return cudaGetLastError();
}

cudaError_t launch_prim_order(const float* sim, int64_t ld, int n, int32_t* rank, int32_t* label, int64_t n_rows,
                              int sms, cudaStream_t stream) {
  if (n < 1 || n > kPrimMax) return cudaErrorInvalidValue;
  prim_order_kernel<<<1, kPrimThreads, 0, stream>>>(sim, ld, n, rank);
  relabel_kernel<<<sms * 4, 256, 0, stream>>>(label, n_rows, rank, n);
  return cudaGetLastError();
}

cudaError_t launch_group_stats(int mode, const void* rows, int64_t row_bytes, int64_t n, int64_t group_rows,
                               int groups, int half_type, void* centres, const PruneStats& st, cudaStream_t stream) {
  const int len = int(mode == kScanHalf ? row_bytes / 2 : row_bytes);
  const size_t smem = size_t(len) * sizeof(float);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(st.top, 0, 4, stream);
  if (e != cudaSuccess) return e;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    kern<<<unsigned(groups), kStatThreads, smem, stream>>>(static_cast<const uint8_t*>(rows), row_bytes, n, group_rows,
                                                           half_type, static_cast<uint8_t*>(centres), st);
    return cudaGetLastError();
  };
  return mode == kScanHalf ? go(group_stats_kernel<false>) : go(group_stats_kernel<true>);
}

cudaError_t launch_prune_lists(int mode, int64_t n, int64_t group_rows, int groups, int64_t ld, const int32_t* U,
                               const float* G, const PruneStats& st, const float* T, int half_len, int32_t* list,
                               int32_t* len, int32_t* block_order, cudaStream_t stream) {
  if (groups < 1 || groups > kPruneGroups) return cudaErrorInvalidValue;
  decide_kernel<<<unsigned(groups), kDecideThreads, 0, stream>>>(mode, n, group_rows, groups, ld, U, G, st, T,
                                                                 half_len, list, len);
  block_order_kernel<<<1, 1024, size_t(groups + 1) * 4, stream>>>(len, groups, (n + BM - 1) / BM,
                                                                  int(group_rows / BM), block_order);
  return cudaGetLastError();
}

}  // namespace evoc
