// 32-bit matrix product on the 5th-generation tensor cores: C[M,N] = A[M,K] * W[N,K]^T with
// float operands taken apart into three bfloat16 terms each (split_utils.cuh).
//
// No precision is given up against the product of plain FP32 multiply-adds (sgemm_f32.cu): of the
// nine products of terms the six that matter are computed, each exact, and the tensor core's sum
// (which cuts instead of rounding) never runs longer than 32 terms of K: the smaller products
// first, then the two steps of the leading terms; each such sum is taken out of tensor memory and
// added in ordinary rounded float, in ascending K.  The reference has no 32-bit product at all:
// every dense product is a cuBLAS bf16 call with float accumulation
// (cuda/kernels/gemm.cu:244-267).
//
// Every output is summed in an order that depends on N, K and the number of products alone, whatever M, the tile or the
// alignment, so a token's result does not depend on which other tokens share the batch.
//
// A CTA computes 128 features x NT token rows over its share of K:
//   warps 0-7    take 32 terms of K of the features apart and store the terms as swizzled tiles
//                into a ring of stages;
//   warps 8-23   take each finished sum out of tensor memory and add;
//   warp 24      issues the products (one elected lane); the warp owns the tensor memory;
//   warp 25      one thread copies the token rows' terms, which a kernel of its own has laid out
//                as the tiles lie in shared memory (up to 16 rows: warps 0-7 do those too);
//   warp 26      one thread fetches the features' floats (TMA) into a ring of its own.  (Rows off
//                the 16-byte boundaries: warps 0-7 read them term by term.)
// Weights of few features have too few tiles for the chip: the CTAs of a cluster (2 or 4, by N, K and the
// number of products alone) then share a tile along K and their sums are added in ascending order through
// distributed shared memory.
//
// Both operands are multiplied by 2^24 before they are taken apart, so that their terms hold floats of every
// size (split_utils.cuh), and the sums by 2^-48.  What is not finite up there shows: infinities, NaN and
// floats from 2^104 on have no terms (one of theirs is a NaN, and so is every sum that they reach); a product
// or a sum beyond 2^80 becomes an infinity or, where a smaller product of terms overflows with a sign of its
// own, a NaN.  So every output whose sum is not finite is computed with multiply-adds in the epilogue,
// one by one.
//
// What bounds it: the warp that issues the products and the shared-memory reads of their
// operands (a step of 32 terms in 0.74 us for 112 token rows, 0.85 for 176; the products alone 0.36
// and 0.56), and waves of tiles that do not fill the chip.  In us against plain multiply-adds:
//   rows x outputs x terms       1      333             2,048
//   4,096 x 2,048        49 -> 24   186 ->  36     797 -> 200
//   2,048 x 2,048        49 -> 15   133 ->  24     409 -> 130
//   12,288 x 2,048       84 -> 43   460 -> 111   2,331 -> 602
// (2,048 rows: 1,030 TFLOP/s of bfloat16 products, at the power limit.)  Without the operands' scaling the last
// line's 333 rows take 109.  Relative error against 64 bits over random
// operands: 0.94e-7 at 2,048 terms and 1.03e-7 at 6,144 (multiply-adds in runs of 64: 1.8e-7, 2.3e-7);
// positive ones: 0.68e-7 and 0.63e-7 (0.82e-7).  On the way here: features' floats into registers instead of by
// TMA 152 us for the third line's 333 rows, products issued from a branch of one lane 122.
#include <cuda.h>

#include "tma_utils.cuh"
#include "umma_utils.cuh"
#include "split_utils.cuh"

namespace {

constexpr int SP_K = 32;                 // terms of K in a stage, and in a tensor-core sum
constexpr int SP_F = 128;                // features of a tile
constexpr int SP_FETCH = 8, SP_SUM = 16;                       // warps
constexpr int SP_MMA = SP_FETCH + SP_SUM, SP_COPY = SP_MMA + 1, SP_TMA = SP_MMA + 2;
constexpr int SP_THREADS = 32 * (SP_TMA + 1);
constexpr int SP_FLOATS = SP_F * SP_K * 4;                     // a stage of the features' floats
constexpr int SP_MAX_FLOATS = 6;                               // such stages
constexpr int SP_MAX_STAGES = 8;
constexpr int SP_RUN = 8;                // sums of a run
constexpr int SP_FEW = 16;               // token rows up to which the product takes them apart itself
constexpr int SP_HEAD = 1024;            // barriers, in front of the ring

struct SplitParams {
  const float *A, *W;
  float* C;
  const uint8_t* terms;                  // of A: [batch][step][term][rows][32], rows of 64 bytes
  long long rows;                        // token rows of a step, whole tiles
  int M, N, K, parts;                    // parts: CTAs that share a tile along K
  int stages, floats;                    // stages of terms; of the features' floats
  long long lda, ldw, ldc, batch_a, batch_w, batch_c;
  int* err;
};

// of: the products side by side in the whole call (which may be cut into several).  From eight on their tiles
// count together: 32 of 512 features and terms for one row took 38.9 us with a cluster of four a
// tile, the multiply-adds 30.7.
int sp_parts(int N, int of) {
  const long long tiles = (long long)((N + SP_F - 1) / SP_F) * (of >= 8 ? of : 1);
  return tiles > 74 ? 1 : tiles > 18 ? 2 : 4;
}

__device__ __forceinline__ uint32_t sp_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void sp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
__device__ __forceinline__ uint32_t sp_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// (x: a multiple of 4 floats)
__device__ __forceinline__ void sp_tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x,
                                               int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ float4 sp_ld4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sp_take(uint32_t taddr, float (&t)[16]) {
  uint32_t r[16];
  tmem_ld16(taddr, r);
#pragma unroll
  for (int i = 0; i < 16; i += 2)
    add2f(t[i], t[i + 1], __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
}
__device__ __forceinline__ void sp_take(uint32_t taddr, float (&t)[8]) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 8; i += 2)
    add2f(t[i], t[i + 1], __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
}
__device__ __forceinline__ void sp_take(uint32_t taddr, float (&t)[4]) {
  uint32_t r[4];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
      : "r"(taddr)
      : "memory");
  add2f(t[0], t[1], __uint_as_float(r[0]), __uint_as_float(r[1]));
  add2f(t[2], t[3], __uint_as_float(r[2]), __uint_as_float(r[3]));
}
// Adds N columns (a multiple of four) onto t, in loads as wide as they go.
template <int N>
__device__ __forceinline__ void sp_add_columns(uint32_t taddr, float* t) {
  if constexpr (N > 0) {
    constexpr int n = N >= 16 ? 16 : N >= 8 ? 8 : 4;
    sp_take(taddr, *reinterpret_cast<float (*)[n]>(t));
    sp_add_columns<N - n>(taddr + n, t + n);
  }
}

// and stores N columns
template <int N>
__device__ __forceinline__ void sp_store_columns(uint32_t taddr, const float* t) {
#pragma unroll
  for (int c = 0; c < N; c += 4)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr + c),
                 "r"(__float_as_uint(t[c])), "r"(__float_as_uint(t[c + 1])),
                 "r"(__float_as_uint(t[c + 2])), "r"(__float_as_uint(t[c + 3]))
                 : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// The plain sum, where that of the terms does not stand for it: in the order of sgemm_f32.cu, ascending
// runs of 64 terms.  (Once NaN, always NaN.)
__device__ __forceinline__ bool sp_finite(float v) { return fabsf(v) < INFINITY; }
template <bool VEC>
__device__ __noinline__ float sp_plain(const float* a, const float* w, int K) {
  float total = 0.f;
  for (int k0 = 0; k0 < K && total == total; k0 += 64) {
    float s = 0.f;
    const int e = min(K, k0 + 64);
    if (VEC) {
#pragma unroll 8
      for (int k = k0; k < e; k += 4) {
        const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s))));
      }
    } else {
#pragma unroll 8
      for (int k = k0; k < e; ++k) s = fmaf(a[k], w[k], s);
    }
    total += s;
  }
  return total;
}

// The terms of A, laid out for the product.  A block takes two rows, four warps to a row.
template <bool VEC>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ A, int M, int K,
                                                         long long lda, long long batch_a,
                                                         uint8_t* __restrict__ terms, long long rows) {
  bf_pdl_trigger();
  const int row = blockIdx.x * 2 + (threadIdx.x >> 7), at = threadIdx.x & 127;
  const int steps = (K + SP_K - 1) / SP_K;
  const float* src = A + blockIdx.z * batch_a + (size_t)min(row, M - 1) * lda;
  uint8_t* dst = terms + (size_t)blockIdx.z * steps * 3 * rows * 64 + (size_t)row * 64 +
                 ((((at & 7) >> 1) ^ ((row >> 1) & 3)) << 4) + ((at & 1) << 3);
  if (row >= M) return;
#pragma unroll 4
  for (int k = 4 * at; k < steps * SP_K; k += 512) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC) {
      if (k < K) v = *reinterpret_cast<const float4*>(src + k);
    } else {
      if (k < K) v.x = src[k];
      if (k + 1 < K) v.y = src[k + 1];
      if (k + 2 < K) v.z = src[k + 2];
      if (k + 3 < K) v.w = src[k + 3];
    }
    uint2 hi, mid, lo;
    split_up(v.x, v.y);
    split_up(v.z, v.w);
    split3(v.x, v.y, hi.x, mid.x, lo.x);
    split3(v.z, v.w, hi.y, mid.y, lo.y);
    uint8_t* to = dst + (size_t)(k / SP_K) * 3 * rows * 64;
    *reinterpret_cast<uint2*>(to) = hi;
    *reinterpret_cast<uint2*>(to + rows * 64) = mid;
    *reinterpret_cast<uint2*>(to + 2 * rows * 64) = lo;
  }
}

// PRE: A's terms come laid out.
template <int NT, bool VEC, bool PRE>
__global__ void __launch_bounds__(SP_THREADS, 1)
sgemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const SplitParams p) {
  // tensor memory: two or three sums; behind them, where a run's sum is added to those of the
  // runs before, KEPT columns of each summing warp (the others stay in registers)
  constexpr int COLS = 512, ACC = NT > 128 ? 2 : 3, KEEP = ACC * NT;
  constexpr int W_BYTES = SP_F * SP_K * 2, A_BYTES = NT * SP_K * 2;      // of one term
  constexpr int STAGE = 3 * (W_BYTES + A_BYTES);
  constexpr int PA = PRE ? 0 : (NT + 31) / 32;                           // pieces of A a thread
  constexpr int MINE = NT / (SP_SUM / 4);                                // columns of a summing warp
  constexpr int KEPT = 4 * ((COLS - KEEP) / 16) < MINE ? 4 * ((COLS - KEEP) / 16) : MINE;
  static_assert(NT % 16 == 0 && NT <= 176, "token rows of a tile");
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(base);
  uint64_t* empty = full + SP_MAX_STAGES;
  uint64_t* acc_full = empty + SP_MAX_STAGES;               // [ACC]
  uint64_t* acc_empty = acc_full + ACC;
  uint64_t* w_full = acc_empty + ACC;
  uint64_t* w_empty = w_full + SP_MAX_FLOATS;
  uint64_t* drain = w_empty + SP_MAX_FLOATS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* tiles = base + SP_HEAD;
  uint8_t* floats = tiles + (size_t)p.stages * STAGE;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int parts = p.parts, rank = parts > 1 ? (int)sp_rank() : 0;
  const int f0 = blockIdx.x / parts * SP_F, m0 = blockIdx.y * NT;
  const float* A = p.A + blockIdx.z * p.batch_a;
  const float* W = p.W + blockIdx.z * p.batch_w;
  float* C = p.C + blockIdx.z * p.batch_c;
  const int steps = (p.K + SP_K - 1) / SP_K;
  const int s0 = (int)((long long)steps * rank / parts), s1 = (int)((long long)steps * (rank + 1) / parts);

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full + s, SP_FETCH + PRE);
      mbar_init(empty + s, 1);
    }
    for (int a = 0; a < ACC; ++a) {
      mbar_init(acc_full + a, 1);
      mbar_init(acc_empty + a, SP_SUM);
    }
    for (int s = 0; s < p.floats; ++s) {
      mbar_init(w_full + s, 1);
      mbar_init(w_empty + s, SP_FETCH);
    }
    mbar_init(drain, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == SP_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  float total[MINE];                       // (summing warps) the columns' sums over K
  int next = 0;                            // (copying threads) the stage that they would fill next,
  uint32_t next_phase = 0;                 // and its phase

  if (warp < SP_FETCH) {
    // ----------------------------------------------------------------- take apart, store
    // 8 threads a row (128 bytes); a thread's rows are 32 apart.  Rows beyond the last count as
    // it, or as zeros: their outputs are not stored.
    const int row = tid >> 3, piece = tid & 7;
    auto get = [&](const float* m, int r, int rows, long long ld, int k) {
      const float* src = m + (size_t)min(r, rows - 1) * ld + k;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (VEC) {
        if (k < p.K) v = *reinterpret_cast<const float4*>(src);
      } else {
        if (k < p.K) v.x = src[0];
        if (k + 1 < p.K) v.y = src[1];
        if (k + 2 < p.K) v.z = src[2];
        if (k + 3 < p.K) v.w = src[3];
      }
      return v;
    };
    const int spot = row * 64 + (((piece >> 1) ^ ((row >> 1) & 3)) << 4) + ((piece & 1) << 3);
    auto put = [&](uint8_t* at, int bytes, float4 v) {
      uint2 hi, mid, lo;
      split_up(v.x, v.y);
      split_up(v.z, v.w);
      split3(v.x, v.y, hi.x, mid.x, lo.x);
      split3(v.z, v.w, hi.y, mid.y, lo.y);
      *reinterpret_cast<uint2*>(at) = hi;
      *reinterpret_cast<uint2*>(at + bytes) = mid;
      *reinterpret_cast<uint2*>(at + 2 * bytes) = lo;
    };
    int stage = 0, slot = 0;
    uint32_t phase = 0, slot_phase = 0;
    float4 wf[4], af[PA + 1];
    auto fetch_a = [&](int s) {
#pragma unroll
      for (int j = 0; j < PA; ++j) af[j] = get(A, m0 + row + 32 * j, p.M, p.lda, s * SP_K + 4 * piece);
    };
    fetch_a(s0);
    for (int s = s0; s < s1; ++s) {
      if (VEC) {
        const bool ok = mbar_wait(w_full + slot, slot_phase, abort);
        if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          wf[j] = *reinterpret_cast<const float4*>(floats + (size_t)slot * SP_FLOATS + j * 4096 + tid * 16);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) wf[j] = get(W, f0 + row + 32 * j, p.N, p.ldw, s * SP_K + 4 * piece);
      }
      const bool ok = mbar_wait(empty + stage, phase ^ 1, abort);
      if (!__all_sync(0xffffffffu, ok)) break;
      uint8_t* at = tiles + (size_t)stage * STAGE + spot;
#pragma unroll
      for (int j = 0; j < 4; ++j) put(at + j * 2048, W_BYTES, wf[j]);
#pragma unroll
      for (int j = 0; j < PA; ++j)
        if (NT % 32 == 0 || j + 1 < PA || row < NT % 32)
          put(at + 3 * W_BYTES + j * 2048, A_BYTES, af[j]);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(full + stage);
        if (VEC) mbar_arrive(w_empty + slot);
      }
      if (PA && s + 1 < s1) fetch_a(s + 1);
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1;
      }
      if (++slot == p.floats) {
        slot = 0;
        slot_phase ^= 1;
      }
    }
  } else if (warp < SP_FETCH + SP_SUM) {
    // ------------------------------------------------------------------------------- sum
    const int quarter = warp & 3, group = (warp - SP_FETCH) >> 2;
    const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(group * MINE);
    const uint32_t kept = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(KEEP + group * KEPT);
    float rest[MINE - KEPT + 1];
#pragma unroll
    for (int i = 0; i < MINE; ++i) total[i] = 0.f;
    int acc = 0;
    uint32_t phase = 0;
    for (int s = s0; s < s1; ++s) {
      const bool ok = mbar_wait(acc_full + acc, phase, abort);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      sp_add_columns<MINE>(at + (uint32_t)(acc * NT), total);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + acc);
      if (++acc == ACC) {
        acc = 0;
        phase ^= 1;
      }
      if ((s - s0) % SP_RUN == SP_RUN - 1 && s + 1 < s1) {     // a run ends
        if (s - s0 >= SP_RUN) {
          sp_add_columns<KEPT>(kept, total);
#pragma unroll
          for (int i = KEPT; i < MINE; ++i) total[i] += rest[i - KEPT];
        }
        sp_store_columns<KEPT>(kept, total);
#pragma unroll
        for (int i = KEPT; i < MINE; ++i) rest[i - KEPT] = total[i];
#pragma unroll
        for (int i = 0; i < MINE; ++i) total[i] = 0.f;
      }
    }
    if (s1 - s0 > SP_RUN && !*abort) {
      sp_add_columns<KEPT>(kept, total);
#pragma unroll
      for (int i = KEPT; i < MINE; ++i) total[i] += rest[i - KEPT];
    }
  } else if (PRE && warp == SP_COPY) {
    // -------------------------------------------------------------- token rows' terms
    bf_pdl_wait();                         // (the kernel that laid them out)
    const uint8_t* src = p.terms + ((size_t)blockIdx.z * steps * 3 * p.rows + m0) * 64;
    if (lane == 0) {
      for (int s = s0; s < s1; ++s) {
        if (!mbar_wait(empty + next, next_phase ^ 1, abort)) break;
        uint8_t* to = tiles + (size_t)next * STAGE + 3 * W_BYTES;
        mbar_expect_tx(full + next, 3 * A_BYTES);
#pragma unroll
        for (int t = 0; t < 3; ++t)
          bf_bulk_load(to + t * A_BYTES, src + ((size_t)s * 3 + t) * p.rows * 64, A_BYTES, full + next);
        if (++next == p.stages) {
          next = 0;
          next_phase ^= 1;
        }
      }
    }
  } else if (VEC && warp == SP_TMA) {
    // ------------------------------------------------------------------ features' floats
    if (lane == 0) {
      for (int s = s0; s < s1; ++s) {
        if (!mbar_wait(w_empty + next, next_phase ^ 1, abort)) break;
        mbar_expect_tx(w_full + next, SP_FLOATS);
        sp_tma_load_3d(floats + (size_t)next * SP_FLOATS, &map_w, w_full + next, s * SP_K, f0,
                       blockIdx.z);
        if (++next == p.floats) {
          next = 0;
          next_phase ^= 1;
        }
      }
    }
  } else if (warp == SP_MMA) {
    // --------------------------------------------------------------------------- products
    const uint64_t desc = umma_desc_k_sw64(smem_u32(tiles));
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NT >> 3) << 17) |
                           ((uint32_t)(SP_F >> 4) << 24);
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    for (int s = s0; s < s1; ++s) {
      const bool ok = mbar_wait(full + stage, phase, abort) && mbar_wait(acc_empty + acc, acc_phase ^ 1, abort);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint64_t wd = desc + (uint64_t)(stage * (STAGE >> 4)), ad = wd + (3 * W_BYTES >> 4);
      const uint32_t d = tmem + (uint32_t)(acc * NT);
      // (term of W, term of A), the smallest products first
      constexpr int TW[6] = {2, 0, 1, 1, 0, 0}, TA[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
      for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int k = 0; k < SP_K / 16; ++k)
          umma_bf16(d, wd + (uint64_t)(TW[t] * (W_BYTES >> 4) + 2 * k),
                    ad + (uint64_t)(TA[t] * (A_BYTES >> 4) + 2 * k), idesc, t > 0 || k > 0);
      umma_commit(empty + stage);
      umma_commit(acc_full + acc);
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1;
      }
      if (++acc == ACC) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  // ----------------------------------------------------------------------------- results
  __syncwarp();
  __syncthreads();
  const int quarter = warp & 3, group = (warp - SP_FETCH) >> 2;
  const bool sums = warp >= SP_FETCH && warp < SP_FETCH + SP_SUM;
  if (*abort) {                            // products still in flight (bounded), then leave
    if (tid == 0) atomicOr(p.err, BF_ERR_WAIT);
    if (warp == SP_MMA) {
      umma_commit(drain);
      const long long t0 = clock64();
      while (!mbar_try_wait(drain, 0) && clock64() - t0 < WAIT_LIMIT_CYCLES / 16) {
      }
    }
    // copies that nobody waited for
    if (PRE && warp == SP_COPY && lane == 0) mbar_drain(full, p.stages, next, next_phase);
    if (VEC && warp == SP_TMA && lane == 0) mbar_drain(w_full, p.floats, next, next_phase);
    __syncwarp();
    __syncthreads();
  }
  if (PRE) bf_pdl_wait();                  // (in every thread, before anything is written)
  if (parts == 1) {
    const int f = f0 + quarter * 32 + lane;
    if (sums && f < p.N) {
      unsigned long long lost = 0;
#pragma unroll
      for (int i = 0; i < MINE; ++i) {
        const int t = group * MINE + i;
        if (m0 + t < p.M) {
          C[(size_t)(m0 + t) * p.ldc + f] = total[i] * (SPLIT_DOWN * SPLIT_DOWN);
          if (!sp_finite(total[i])) lost |= 1ull << i;
        }
      }
      for (; lost; lost &= lost - 1) {
        const int t = m0 + group * MINE + __ffsll(lost) - 1;
        C[(size_t)t * p.ldc + f] = sp_plain<VEC>(A + (size_t)t * p.lda, W + (size_t)f * p.ldw, p.K);
      }
    }
  } else {
    // (the ring is free: every product is complete)  [token][feature], read by the ranks in turn
    float* mine = reinterpret_cast<float*>(tiles);
    if (sums) {
#pragma unroll
      for (int i = 0; i < MINE; ++i) mine[(group * MINE + i) * SP_F + quarter * 32 + lane] = total[i];
    }
    sp_cluster_sync();
    const uint32_t mine_at = smem_u32(mine);
    const int f = f0 + 4 * lane;
    const bool vec = f + 4 <= p.N && (p.ldc & 3) == 0 && ((uintptr_t)C & 15) == 0;
    if (warp < SP_FETCH + SP_SUM) {
      for (int t = rank + parts * warp; t < NT && m0 + t < p.M; t += parts * (SP_FETCH + SP_SUM)) {
        const uint32_t at = mine_at + (uint32_t)((t * SP_F + 4 * lane) * 4);
        float4 v = sp_ld4(sp_map(at, 0));
        for (int r = 1; r < parts; ++r) {
          const float4 u = sp_ld4(sp_map(at, r));
          v.x += u.x;
          v.y += u.y;
          v.z += u.z;
          v.w += u.w;
        }
        float* e[4] = {&v.x, &v.y, &v.z, &v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) *e[j] *= SPLIT_DOWN * SPLIT_DOWN;
        if (!(sp_finite(v.x) && sp_finite(v.y) && sp_finite(v.z) && sp_finite(v.w))) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (!sp_finite(*e[j]) && f + j < p.N)
              *e[j] = sp_plain<VEC>(A + (size_t)(m0 + t) * p.lda, W + (size_t)(f + j) * p.ldw, p.K);
        }
        float* dst = C + (size_t)(m0 + t) * p.ldc + f;
        if (vec) {
          *reinterpret_cast<float4*>(dst) = v;
        } else {
          if (f < p.N) dst[0] = v.x;
          if (f + 1 < p.N) dst[1] = v.y;
          if (f + 2 < p.N) dst[2] = v.z;
          if (f + 3 < p.N) dst[3] = v.w;
        }
      }
    }
    sp_cluster_sync();                     // (a peer may still read this CTA's sums)
  }
  __syncthreads();
  if (warp == SP_MMA) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS)
                 : "memory");
  }
}

template <int NT, bool VEC>
int sp_launch(const CUtensorMap& map, SplitParams p, int batch, uint8_t* scratch, cudaStream_t stream) {
  constexpr bool PRE = NT > SP_FEW;
  constexpr int STAGE = 3 * (SP_F + NT) * SP_K * 2;
  constexpr int room = 226 * 1024 - 1024 - SP_HEAD;
  constexpr int stages = (room - 3 * SP_FLOATS) / STAGE < SP_MAX_STAGES ? (room - 3 * SP_FLOATS) / STAGE
                                                                       : SP_MAX_STAGES;
  constexpr int left = (room - stages * STAGE) / SP_FLOATS;
  static_assert(stages >= 2 && left >= 3, "room for the rings");
  p.stages = stages;
  p.floats = left < SP_MAX_FLOATS ? left : SP_MAX_FLOATS;
  size_t smem = 1024 + SP_HEAD + (size_t)p.stages * STAGE + (size_t)p.floats * SP_FLOATS;
  // one CTA an SM: two that hold tensor memory and wait for their clusters could wait for each other
  if (smem < 120 * 1024) smem = 120 * 1024;
  auto kern = sgemm_split_kernel<NT, VEC, PRE>;
  static bool configured_on[BF_MAX_DEVICES];
  bool& configured = configured_on[bf_current_device()];
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int tiles = (p.M + NT - 1) / NT;
  if (PRE) {
    p.rows = (long long)tiles * NT;
    p.terms = scratch;
    split_rows_kernel<VEC><<<dim3((p.M + 1) / 2, 1, batch), 256, 0, stream>>>(
        p.A, p.M, p.K, p.lda, p.batch_a, scratch, p.rows);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.N + SP_F - 1) / SP_F * p.parts), tiles, batch);
  cfg.blockDim = SP_THREADS;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = bf_pdl_enabled();
  cfg.attrs = attr;
  cfg.numAttrs = PRE ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map, p);
  return e != cudaSuccess ? (int)e : bf_launch_status();
}

// Token rows of a tile.
int sp_tile(int M, int N, int batch, int of) {
  const long long cols = (long long)((N + SP_F - 1) / SP_F) * sp_parts(N, of) * batch;
  if (M <= SP_FEW) return SP_FEW;
  // a step of K took 0.74 us in tiles of 112 rows and 0.85 in tiles of 176 (one tile an SM)
  auto waves = [&](int n) { return (cols * ((M + n - 1) / n) + 147) / 148; };
  return waves(112) * 74 <= waves(176) * 85 ? 112 : 176;
}

}  // namespace

// Bytes of scratch that bf_sgemm_split needs for these sizes (may be 0).
BF_EXPORT long long bf_sgemm_split_scratch(int M, int N, int K, int batch, int of, int nt) {
  if (M <= SP_FEW) return 0;
  if (!nt) nt = sp_tile(M, N, batch, of);
  const long long rows = (long long)((M + nt - 1) / nt) * nt, steps = (K + SP_K - 1) / SP_K;
  return batch * steps * 3 * rows * 64;
}

// C[M, N] = A[M, K] * W[N, K]^T, `batch` of them (bf_sgemm_nt_batched's strides), of `of` that the
// caller has (the order of sums depends on those).  nt: token rows of a tile (0: chosen here).  M up to
// 65,535 tiles.
BF_EXPORT int bf_sgemm_split(const float* A, const float* W, float* C, int M, int N, int K,
                             long long lda, long long ldw, long long ldc, int batch, int of,
                             long long batch_a, long long batch_w, long long batch_c, int nt,
                             void* scratch, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (!nt) nt = sp_tile(M, N, batch, of);
  if (K <= 0 || batch > 65535 || (M + nt - 1) / nt > 65535 || ((uintptr_t)scratch & 15) ||
      (nt > SP_FEW && !scratch))
    return (int)cudaErrorInvalidValue;
  SplitParams p = {A, W, C, nullptr, 0, M, N, K, K < 512 ? 1 : sp_parts(N, of), 0, 0, lda, ldw, ldc,
                   batch_a, batch_w, batch_c, err};
  CUtensorMap map = {};
  bool vec = ((K | lda | ldw | batch_a | batch_w) & 3) == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 &&
             ldw > 0 && (batch == 1 || batch_w > 0);
  if (vec) {
    BfEncodeTiledFn enc = bf_encode_tiled();
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)N, (cuuint64_t)batch};
    const cuuint64_t strides[2] = {(cuuint64_t)ldw * 4, (cuuint64_t)(batch == 1 ? ldw : batch_w) * 4};
    const cuuint32_t box[3] = {SP_K, SP_F, 1}, estr[3] = {1, 1, 1};
    vec = enc && enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(W), dims, strides, box,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
#define SP_GO(n)                                                       \
  return vec ? sp_launch<n, true>(map, p, batch, (uint8_t*)scratch, stream) \
             : sp_launch<n, false>(map, p, batch, (uint8_t*)scratch, stream)
  switch (nt) {
    case 16: SP_GO(16);
    case 112: SP_GO(112);
    case 176: SP_GO(176);
  }
#undef SP_GO
  return (int)cudaErrorInvalidValue;
}
