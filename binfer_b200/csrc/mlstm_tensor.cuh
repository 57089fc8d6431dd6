// The products of the matrix memory's chunks (chunk_scan.cu) on the 5th-generation tensor cores: q, k and v are
// bfloat16 numbers, states, weights and weighted values floats in three bfloat16 terms (split_utils.cuh).
//
//   mt_state   cs_state and cs_prefix in one: a CTA keeps 64 x 128 elements of a head's state in
//              registers and goes from chunk to chunk.  The states between the chunks are written
//              once (before: what a chunk adds written, read, the state written in its place)
//   mt_out     cs_out: 64 tokens x 128 value sizes a tile; a CTA an SM goes from tile to tile
//
// Both are a stream of steps of 64 (tokens of a chunk, or key sizes).  Sixteen warps fetch a step's
// operands a step ahead (into shared memory: held in registers they were
// spilled, and a spill waits for its load), weight them, take them apart and store the terms; a
// seventeenth issues the products; while they run the sixteen take the sums of the step before
// out of tensor memory and add.
//
// A product of a float and a bfloat16 number is three products of terms.  The tensor core's sums cut
// where arithmetic rounds, so the leading terms' products are summed 32 at a time, apart from the
// smaller terms', and the sums are added in rounded float.  Floats are multiplied by 2^24 before they are
// taken apart, so that their terms hold them whatever their size (split_utils.cuh), and the sums by 2^-24.
// Operands that have no terms (infinities, NaN, floats from 2^104 on) are zero in the products, and the
// results that they reach are computed by multiply-adds; so are sums that are not finite (where finite
// operands' product leaves float's range, that of a smaller term may overflow with a sign of its own).
//
// 2,048 tokens, 8 heads of 256 x 512: mt_state 73 us (cs_state and cs_prefix 177), mt_out 91 (cs_out 168).
// What bounds them: mt_state the issue slots (a chunk's keys and values to take apart, its sums, its states
// to store: some 4,000 cycles for 600 of products), mt_out the same (a step 2,500 cycles) and the start
// and the end of a tile (4,000).  Relative errors against 64 bits, this / those, at 2,048 tokens (four inputs):
// outputs 5.7 7.1 6.4 5.5 / 5.5 8.8 7.5 5.8 e-7, states 0.85 1.2 0.94 0.98 / 1.4 1.5 1.4 1.3 e-7.
//
// The recurrences whose operands are floats have kernels of their own (chunk_tensor.cuh): with six products and
// both operands to take apart these took 90 + 144 us where multiply-adds took 188 (2,000 tokens, 64 heads of 128 x 64).
//
// Included by chunk_scan.cu behind its helpers.
#pragma once
#include "split_utils.cuh"
#include "tma_utils.cuh"

#define MT_C 64            // tokens of a chunk, and sizes of a step
#define MT_M 128           // value sizes of a tile: the products' rows
#define MT_WORK 512        // threads that take apart and add
#define MT_THREADS (MT_WORK + 32)
#define MT_MMA (MT_WORK / 32)
#define MT_TILE (MT_M * MT_C * 2)              // bytes of a term of the products' rows
#define MT_TOK (MT_C * MT_C * 2)               // and of their columns
#define MT_COLS 512                            // tensor memory: two places of 3 x 64 columns

typedef __nv_bfloat16 mt_bf16;

// Eight columns of three places of tensor memory, 64 columns from one to the next: the sums of the leading
// terms' two halves and the others', added up
__device__ __forceinline__ void mt_take(uint32_t at, unsigned long long (&u)[4]) {
  uint32_t r[24];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%25];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%26];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23])
      : "r"(at), "r"(at + MT_C), "r"(at + 2 * MT_C)
      : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    unsigned long long x[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      x[k] = cs_pair(__uint_as_float(r[8 * k + 2 * i]), __uint_as_float(r[8 * k + 2 * i + 1]));
    u[i] = cs_add2(cs_add2(x[0], x[1]), x[2]);
  }
}

__device__ __forceinline__ unsigned long long mt_down(unsigned long long x) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(cs_pair(SPLIT_DOWN, SPLIT_DOWN)));
  return r;
}

// Sixteen bytes on their way into shared memory
__device__ __forceinline__ void mt_fetch(uint8_t* to, const void* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to)), "l"(from));
}
__device__ __forceinline__ void mt_fetched() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Eight numbers: two float4, or bfloat16 as they lie
struct MtEight {
  float v[8];
};
__device__ __forceinline__ MtEight mt_bf16s(const uint4& u) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  MtEight x;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x.v[2 * i] = __uint_as_float(w[i] << 16);
    x.v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
  return x;
}
// Their terms, times SPLIT_UP, to `at`, a term's tile `bytes` behind the one before.  `left` stays finite
// where all have terms.
__device__ __forceinline__ void mt_put(uint8_t* at, int bytes, MtEight x, float2& left) {
  uint4 hi, mid, lo;
#pragma unroll
  for (int i = 0; i < 8; i += 2) split_up(x.v[i], x.v[i + 1]);
  split3(x.v[0], x.v[1], hi.x, mid.x, lo.x, left);
  split3(x.v[2], x.v[3], hi.y, mid.y, lo.y, left);
  split3(x.v[4], x.v[5], hi.z, mid.z, lo.z, left);
  split3(x.v[6], x.v[7], hi.w, mid.w, lo.w, left);
  *reinterpret_cast<uint4*>(at) = hi;
  *reinterpret_cast<uint4*>(at + bytes) = mid;
  *reinterpret_cast<uint4*>(at + 2 * bytes) = lo;
}
__device__ __forceinline__ bool mt_bad(const float2& left) { return !(fabsf(left.x + left.y) < INFINITY); }
// an infinity or a NaN among eight bfloat16 numbers
__device__ __forceinline__ bool mt_bad(const uint4& u) {
  auto two = [](uint32_t w) { return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u; };
  return two(u.x) || two(u.y) || two(u.z) || two(u.w);
}
// zero in the place of what has no terms: a bit for each.  What is an infinity or a NaN among bfloat16
// numbers; among floats what is beyond the largest of those once it is multiplied.
constexpr uint32_t MT_NO_TERMS = 0x7f7f8000u, MT_NO_TERMS_UP = MT_NO_TERMS - (24u << 23);
__device__ __forceinline__ int mt_clean(MtEight& x, uint32_t from) {
  int bad = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((__float_as_uint(x.v[i]) & 0x7fffffffu) >= from) {
      bad |= 1 << i;
      x.v[i] = 0.f;
    }
  return bad;
}
__device__ __forceinline__ uint4 mt_pack(const MtEight& x) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    w[i] = __byte_perm(__float_as_uint(x.v[2 * i]), __float_as_uint(x.v[2 * i + 1]), 0x7632);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Where a piece of eight goes: rows of 128 bytes (64 numbers), 128-byte swizzle.  K-major: row =
// row of the product.  MN-major: row = K, 64 of the product's rows side by side, blocks of those
// behind one another.
__device__ __forceinline__ int mt_spot(int row, int piece) { return row * 128 + ((piece ^ (row & 7)) << 4); }
__device__ __forceinline__ int mt_spot_mn(int k, int piece) {
  return (piece >> 3) * (MT_C * 128) + mt_spot(k, piece & 7);
}

// The products of a step by a converged warp: rows' terms (TA, MN-major) times columns' (TB), 64 columns; the
// first and the second 64 columns of `d` take the leading terms' first and second 32, the next the rest.
template <int TA, int TB, bool B_MN>
__device__ __forceinline__ void mt_products(uint32_t d, uint32_t a, uint32_t b) {
  constexpr int ka = 16 * 128, kb = B_MN ? 16 * 128 : 32;      // 16 terms further
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((uint32_t)B_MN << 16) |
                         ((uint32_t)(MT_C >> 3) << 17) | ((uint32_t)(MT_M >> 4) << 24);
  const uint64_t da = umma_desc_mn_sw128(a, MT_C * 128);
  const uint64_t db = B_MN ? umma_desc_mn_sw128(b, MT_C * 128) : umma_desc_k_sw128(b);
#pragma unroll
  for (int t = 2; t > 0; --t)                    // (one side has one term) the smallest first
#pragma unroll
    for (int k = 0; k < 4; ++k)
      umma_bf16(d + 2 * MT_C, da + (uint64_t)(((TA > 1 ? t : 0) * MT_TILE + k * ka) >> 4),
                     db + (uint64_t)(((TB > 1 ? t : 0) * MT_TOK + k * kb) >> 4), idesc, t < 2 || k > 0);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    umma_bf16(d + (k >> 1) * MT_C, da + (uint64_t)(k * ka >> 4), db + (uint64_t)(k * kb >> 4), idesc, k & 1);
}

struct MtShared {
  uint64_t done[2], drain, got[2];  // a step's products are complete (even and odd steps); all are; a copy is here
  uint32_t tmem;
  int abort;
};
__device__ __forceinline__ uint32_t mt_begin(MtShared& s) {
  if (threadIdx.x == 0) {
    mbar_init(s.done, 1);
    mbar_init(s.done + 1, 1);
    mbar_init(&s.drain, 1);
    mbar_init(s.got, 1);
    mbar_init(s.got + 1, 1);
    s.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x >> 5 == MT_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s.tmem)),
                 "r"(MT_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return s.tmem;
}
__device__ __forceinline__ void mt_end(MtShared& s, uint32_t tmem, int* err) {
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (*(volatile int*)&s.abort) {                        // (a wait gave up)
    if (threadIdx.x == 0) atomicOr(err, BF_ERR_WAIT);
    if (threadIdx.x >> 5 == MT_MMA) {                    // products still in flight
      umma_commit(&s.drain);
      const long long t0 = clock64();
      while (!mbar_try_wait(&s.drain, 0) && clock64() - t0 < WAIT_LIMIT_CYCLES / 16) {
      }
    }
    __syncwarp();
    __syncthreads();
  }
  if (threadIdx.x >> 5 == MT_MMA) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MT_COLS)
                 : "memory");
  }
}
// A step's terms are stored, by all threads, and what they took out of tensor memory is taken.
__device__ __forceinline__ void mt_stored() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
}
// Step `i`'s products are complete.  (When a wait gives up the kernel goes on, without waits and without
// further copies into shared memory, to its end.)
__device__ __forceinline__ void mt_done(MtShared& s, int i) {
  mbar_wait(s.done + (i & 1), (i >> 1) & 1, &s.abort);
  __syncwarp();
  tc_fence_after();
}

// --------------------------------------------------------------------------------- mt_state
// grid (tiles of 64 key x 128 value sizes of a head's state, H, B); n, by the first tiles of values.  The state lies as
// [dk][dv]; the products' rows are value sizes, so that what the lanes of a warp hold lies side by
// side.  Between the chunks (U): [dv / 128][dk][128], so that a CTA's elements are one block, which
// leaves through shared memory in one copy (16 stores a thread held the kernel at 163 us).
#define MT_STATE_STAGE (3 * MT_TILE + MT_TOK)
#define MT_STATE_SMEM (1024 + 2 * MT_STATE_STAGE + MT_WORK * 48 + 2 * MT_C * MT_M * 4)
__global__ void __launch_bounds__(MT_THREADS, 1) mt_state_kernel(
    const mt_bf16* __restrict__ proj, CsIn p, const int* __restrict__ q_start,
    float* __restrict__ state, long long slot_stride, int state_size,
    const int* __restrict__ state_slots, int n_slots, const double* __restrict__ G,
    const double* __restrict__ g0, const float2* __restrict__ Wl, float* __restrict__ U,
    float* __restrict__ Un, int* __restrict__ err) {
  extern __shared__ __align__(16) uint8_t mt_raw[];
  __shared__ MtShared sh;
  __shared__ int odd, odd_v[3][MT_M], odd_k[3][MT_C];   // (of chunk % 3) the last chunk with a size that has no terms
  __shared__ __align__(16) float2 w_s[4][MT_C];         // (of chunk % 4) the tokens' weights
  __shared__ float n_s[3][MT_WORK / 32][MT_C];          // (of chunk % 3) the warps' shares of the weighted keys' sum
  uint8_t* tiles = mt_raw + ((1024u - (smem_u32(mt_raw) & 1023u)) & 1023u);
  const int h = blockIdx.y, b = blockIdx.z;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, 0, b);
  if (c.n <= p.n_min) return;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= n_slots) {
    if (threadIdx.x == 0) atomicOr(err, BF_ERR_SLOT);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const mt_bf16* kp = proj + (size_t)c.t0 * p.qk_stride + p.k_off + (size_t)h * p.dk;
  const mt_bf16* vp = proj + (size_t)c.t0 * p.v_stride + p.v_off + (size_t)h * p.dv;
  const float2* wl = Wl + (size_t)h * p.T + c.t0;
  const double* g = G + (size_t)h * p.T + c.t0;
  const int chunks = (c.n + MT_C - 1) / MT_C, tiles_k = p.dk / MT_C;
  float* st = state + (size_t)slot * slot_stride + (size_t)h * state_size;
  const double first = g0[(size_t)b * p.H + h];
  auto decay = [&](int i) {                      // over chunk i
    return cs_exp(g[min(c.n, (i + 1) * MT_C) - 1] - (i ? g[i * MT_C - 1] : first));
  };

  const int k0 = (int)blockIdx.x % tiles_k * MT_C, v0 = (int)blockIdx.x / tiles_k * MT_M;
  for (int i = tid; i < 3 * MT_M; i += MT_THREADS) odd_v[i / MT_M][i % MT_M] = -1;
  if (tid < 3 * MT_C) odd_k[tid / MT_C][tid % MT_C] = -1;
  if (tid == 0) odd = 0;
  if (tid < 2 * MT_C && tid < c.n) w_s[tid / MT_C][tid % MT_C] = wl[tid];
  const uint32_t tmem = mt_begin(sh);

  if (warp == MT_MMA) {
    for (int i = 0; i < chunks; ++i) {
      mt_stored();
      tc_fence_after();
      const uint32_t at = smem_u32(tiles) + (uint32_t)((i & 1) * MT_STATE_STAGE);
      mt_products<3, 1, true>(tmem + (uint32_t)((i & 1) * 3 * MT_C), at, at + 3 * MT_TILE);
      umma_commit(sh.done + (i & 1));
    }
    mt_end(sh, tmem, err);
    return;
  }

  // ---- operands: two pieces of v a thread (rows 32 apart), one of k; the weights, two chunks ahead.
  // Rows beyond the last repeat it and count as zeros.
  const int vq = tid & 15, vr = tid >> 4, kq = tid & 7, kr = tid >> 3;
  uint8_t* mine = tiles + 2 * MT_STATE_STAGE + tid * 16;
  auto fetch = [&](int i) {
    const int a = i * MT_C, last = c.n - 1;
    mt_fetch(mine, vp + (size_t)min(a + vr, last) * p.v_stride + v0 + 8 * vq);
    mt_fetch(mine + 16 * MT_WORK, vp + (size_t)min(a + vr + 32, last) * p.v_stride + v0 + 8 * vq);
    mt_fetch(mine + 32 * MT_WORK, kp + (size_t)min(a + kr, last) * p.qk_stride + k0 + 8 * kq);
    if (tid < MT_C && a + MT_C + tid < c.n) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(&w_s[(i + 1) & 3][tid])),
                   "l"(wl + a + MT_C + tid));
    }
  };
  auto value = [&](int i, int x) {               // weighted
    MtEight e = {};
    const int s = vr + 32 * x;
    if (i * MT_C + s >= c.n) return e;
    e = mt_bf16s(*reinterpret_cast<const uint4*>(mine + x * 16 * MT_WORK));
    const float2 w = w_s[i & 3][s];
#pragma unroll
    for (int j = 0; j < 8; ++j) e.v[j] = cs_times(e.v[j], w);
    return e;
  };
  const int v_spot = mt_spot_mn(vr, vq), k_spot = 3 * MT_TILE + mt_spot(kr, kq);
  auto convert = [&](int i) {
    uint8_t* tile = tiles + (i & 1) * MT_STATE_STAGE;
    mt_fetched();
    float2 left = make_float2(0.f, 0.f);
#pragma unroll
    for (int x = 0; x < 2; ++x) mt_put(tile + v_spot + x * 4096, MT_TILE, value(i, x), left);
    uint4 k = *reinterpret_cast<const uint4*>(mine + 32 * MT_WORK);
    if (i * MT_C + kr >= c.n) k = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4*>(tile + k_spot) = k;
    if (v0 == 0) {                               // n's share: this warp's four tokens
      MtEight e = mt_bf16s(k);
      const float2 w = i * MT_C + kr < c.n ? w_s[i & 3][kr] : make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        e.v[j] = cs_times(e.v[j], w);
        e.v[j] += __shfl_xor_sync(0xffffffffu, e.v[j], 8);
        e.v[j] += __shfl_xor_sync(0xffffffffu, e.v[j], 16);
      }
      if (lane < 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) n_s[i % 3][warp][8 * lane + j] = e.v[j];
      }
    }
    if (mt_bad(left) || mt_bad(k)) {
#pragma unroll 1
      for (int x = 0; x < 3; ++x) {
        MtEight e = x < 2 ? value(i, x) : mt_bf16s(k);
        const int bad = mt_clean(e, x < 2 ? MT_NO_TERMS_UP : MT_NO_TERMS);
        for (int j = 0; j < 8; ++j)
          if (bad >> j & 1) (x < 2 ? odd_v[i % 3] + 8 * vq : odd_k[i % 3] + 8 * kq)[j] = i;
        if (x < 2) mt_put(tile + v_spot + x * 4096, MT_TILE, e, left);
        else *reinterpret_cast<uint4*>(tile + k_spot) = mt_pack(e);
      }
      odd = 1;
    }
  };

  // ---- the state: value size v0 + 32 quarter + lane, key sizes k0 + 16 group ..
  const int quarter = warp & 3, group = warp >> 2;
  const int v_own = quarter * 32 + lane;
  const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(group * 16);
  float* own = st + (size_t)(k0 + group * 16) * p.dv + v0 + v_own;
  float* kept = reinterpret_cast<float*>(tiles + 2 * MT_STATE_STAGE + MT_WORK * 48);       // [2][64][128]
  float* mine_kept = kept + group * 16 * MT_M + v_own;
  // (by one thread, once all have written the state before chunk i)
  auto send = [&](int i) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                     U + ((size_t)(c.first + i) * p.H + h) * p.dk * p.dv + (size_t)v0 * p.dk + k0 * MT_M),
                 "r"(smem_u32(kept + (i & 1) * MT_C * MT_M)), "r"(MT_C * MT_M * 4)
                 : "memory");
    bf_bulk_commit();
  };
  unsigned long long S[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) S[j] = cs_pair(own[(size_t)(2 * j) * p.dv], own[(size_t)(2 * j + 1) * p.dv]);
  float2 dec = make_float2(0.f, 0.f);            // (lane l: over chunk l of the current 32)
  const bool has_n = v0 == 0 && tid < MT_C;
  float* n_at = st + p.dk * p.dv + k0 + tid;
  float n_own = has_n ? *n_at : 0.f;
  auto finish = [&](int i) {
    if ((i & 31) == 0) dec = decay(min(i + lane, chunks - 1));
    const float dx = __shfl_sync(0xffffffffu, dec.x, i & 31), dy = __shfl_sync(0xffffffffu, dec.y, i & 31);
    if (has_n) {
      float x[MT_WORK / 32];
#pragma unroll
      for (int j = 0; j < MT_WORK / 32; ++j) x[j] = n_s[i % 3][j][tid];
#pragma unroll
      for (int o = MT_WORK / 64; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < o; ++j) x[j] += x[j + o];
      Un[((size_t)(c.first + i) * p.H + h) * p.dk + k0 + tid] = n_own;
      n_own = fmaf(dx, n_own, fmaf(dy, n_own, x[0]));
    }
    const unsigned long long dx2 = cs_pair(dx, dx), dy2 = cs_pair(dy, dy);
    float* to = mine_kept + (i & 1) * MT_C * MT_M;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float a, e;
      cs_unpair(S[j], a, e);
      to[2 * j * MT_M] = a;
      to[(2 * j + 1) * MT_M] = e;
    }
    mt_done(sh, i);
    unsigned long long zero = 0ull;              // (NaN where some sum is not finite)
#pragma unroll
    for (int j0 = 0; j0 < 8; j0 += 4) {
      unsigned long long u[4];
      mt_take(at + (uint32_t)((i & 1) * 3 * MT_C + 2 * j0), u);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        S[j0 + j] = cs_fma2(dx2, S[j0 + j], cs_fma2(dy2, S[j0 + j], mt_down(u[j])));
        zero = cs_fma2(u[j], 0ull, zero);
      }
    }
    float z0, z1;
    cs_unpair(zero, z0, z1);
    const bool lost = z0 + z1 != 0.f;
    if (odd || lost) {
#pragma unroll 1
      for (int j = 0; j < 16; ++j) {
        float now = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float a, x;
          cs_unpair(S[k], a, x);
          now = 2 * k == j ? a : 2 * k + 1 == j ? x : now;
        }
        if (odd_v[i % 3][v_own] != i && odd_k[i % 3][group * 16 + j] != i &&
            !(lost && !(fabsf(now) < INFINITY)))
          continue;
        const int e = min(c.n, (i + 1) * MT_C);
        float y = 0.f;                           // the chunk's share by multiply-adds
#pragma unroll 1
        for (int s = i * MT_C; s < e; ++s)
          y = fmaf(bf_ld(kp + (size_t)s * p.qk_stride + k0 + group * 16 + j),
                   cs_times(bf_ld(vp + (size_t)s * p.v_stride + v0 + v_own), wl[s]), y);
        const float was = to[j * MT_M], is = fmaf(dx, was, fmaf(dy, was, y));
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float a, x;
          cs_unpair(S[k], a, x);
          S[k] = cs_pair(2 * k == j ? is : a, 2 * k + 1 == j ? is : x);
        }
      }
    }
  };

  fetch(0);
  for (int i = 0; i < chunks; ++i) {
    convert(i);                    // (the products that read this stage are complete: finish(i - 2))
    if (tid == 0) bf_bulk_wait_read<0>();        // (finish(i - 1) writes the place of the last copy)
    mt_stored();
    if (tid == 0 && i > 1) send(i - 2);
    fetch(min(i + 1, chunks - 1));
    if (i) finish(i - 1);
  }
  if (tid == 0) bf_bulk_wait_read<0>();
  asm volatile("barrier.cta.sync 1, %0;" ::"n"(MT_WORK) : "memory");
  finish(chunks - 1);
  if (has_n) *n_at = n_own;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("barrier.cta.sync 1, %0;" ::"n"(MT_WORK) : "memory");
  if (tid == 0) {
    if (chunks > 1) send(chunks - 2);
    send(chunks - 1);
    bf_bulk_wait_read<0>();
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) cs_unpair(S[j], own[(size_t)(2 * j) * p.dv], own[(size_t)(2 * j + 1) * p.dv]);
  mt_fetched();
  mt_end(sh, tmem, err);
}

// ----------------------------------------------------------------------------------- mt_out
// Tiles of (chunk, head, 128 value sizes), dealt out to a CTA an SM.  The products' rows are value
// sizes, their columns the chunk's tokens: first the state times q over dk, a step of 64 at a time,
// times the token's weight, then the values times the weighted q . k.
//
// The weights inside a chunk, exp(G_t - H_s): where s lies in an earlier block of 16 tokens than t,
// with the block's last G between them, exp(G_t - G) exp(G - H_s), each factor (at most 1) a float and
// what is left of it; the exponentials of a chunk are so some 700 instead of 2,080.
struct MtUnit {                  // a tile: value sizes m0 .., head, chunk, request (-1: none), the chunk's first token,
  int m0, h, chunk, b, t0, n, index;   // its tokens, its number in the request
};
struct MtTable {                 // of a tile
  MtUnit unit;
  double g[MT_C], h[MT_C];
  float2 at[MT_C];               // the token's weight of the state before the chunk (times q_scale)
  float2 row[3][MT_C], col[48];  // exp(G_t - G of block b's end); exp(that - H_s)
  float2 near[MT_C][16];         // exp(G_t - H_s) inside a block
  float den[MT_C];
  int odd_t[MT_C], odd_m[MT_M], odd;   // the token's operands have no terms; from which token on the row's
};                                     // some have none; any
// a stage: the rows' three terms and q (one term), or the values (one term) and q . k in three; what a step's
// operands are made from, for two steps (with one place, asked for behind the step before, 95 us; so 91)
#define MT_OUT_STAGE (3 * MT_TILE + MT_TOK)
#define MT_OUT_RAW (MT_C * MT_M * 4 + MT_WORK * 16)
#define MT_OUT_SMEM (1024 + 2 * MT_OUT_STAGE + 2 * MT_OUT_RAW)
__global__ void __launch_bounds__(MT_THREADS, 1) mt_out_kernel(
    const mt_bf16* __restrict__ proj, CsIn p, int n_chunks, const int* __restrict__ q_start,
    const int* __restrict__ state_slots, int n_slots, const double* __restrict__ G,
    const double* __restrict__ Hs, const double* __restrict__ g0, const float* __restrict__ E,
    const float* __restrict__ qkm, const float* __restrict__ U, const float* __restrict__ Un,
    float* __restrict__ o_raw, int* __restrict__ err) {
  extern __shared__ __align__(16) uint8_t mt_raw[];
  __shared__ MtShared sh;
  __shared__ MtTable table[2];
  __shared__ MtUnit next_s;                      // the tile after the one in work, found by the issuing warp
  __shared__ __align__(16) float n_s[2][MT_C];   // n's sizes of the step
  uint8_t* ring = mt_raw + ((1024u - (smem_u32(mt_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m_tiles = p.dv / MT_M, steps = p.dk / MT_C;
  const int units = n_chunks * p.H * m_tiles;
  const uint32_t tmem = mt_begin(sh);

  // tiles of a chunk and head follow one another, so that the CTAs which share them run together
  auto unit_at = [&](int u) {
    MtUnit x;
    x.m0 = u % m_tiles * MT_M;
    x.h = u / m_tiles % p.H;
    x.chunk = u / (m_tiles * p.H);
    const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, x.chunk, -1);
    const int slot = c.b < 0 ? -1 : state_slots[c.b];
    x.b = slot < 0 || slot >= n_slots ? -1 : c.b;
    x.index = c.index;
    x.t0 = c.t0 + c.index * MT_C;
    x.n = min(MT_C, c.n - c.index * MT_C);
    return x;
  };

  if (warp == MT_MMA) {
    int u = blockIdx.x;
    auto next = [&]() {                          // (b < 0: none)
      MtUnit x = {0, 0, 0, -1, 0, 0, 0};
      for (; u < units && x.b < 0; u += gridDim.x) x = unit_at(u);
      if (lane == 0) next_s = x;
      return x.b >= 0;
    };
    bool more = next();
    __syncthreads();
    for (int i = 0; more;) {
      __syncthreads();                           // (the tile's tables)
      for (int step = 0; step <= steps; ++step, ++i) {
        mt_stored();
        tc_fence_after();
        const uint32_t tm = smem_u32(ring) + (uint32_t)((i & 1) * MT_OUT_STAGE);
        const uint32_t d = tmem + (uint32_t)((i & 1) * 3 * MT_C);
        if (step < steps) mt_products<3, 1, false>(d, tm, tm + 3 * MT_TILE);
        else mt_products<1, 3, false>(d, tm, tm + MT_TILE);
        umma_commit(sh.done + (i & 1));
        if (step == 0) more = next();            // (read by the others behind a later step's barrier)
      }
    }
    mt_end(sh, tmem, err);
    return;
  }

  const int tq = tid & 7, tr = tid >> 3;         // token operand: row tr, sizes 8 tq ..
  const int mq = tid & 15, mr = tid >> 4;        // rows of value sizes: K rows mr, mr + 32, sizes 8 mq ..
  const int t_spot = mt_spot(tr, tq), m_spot = mt_spot_mn(mr, mq);
  const int quarter = warp & 3, group = warp >> 2;                       // results: tokens 16 group ..
  const int m = quarter * 32 + lane;
  const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(group * 16);
  // a step's floats (the state's 64 rows of 128, or q . k) come in one copy, q's or the values' rows in
  // pieces of sixteen bytes that the same thread reads behind them
  uint8_t* block = ring + 2 * MT_OUT_STAGE;
  auto place = [&](int i) { return block + (i & 1) * MT_OUT_RAW; };
  auto eight = [&](int i, int row, int width, int piece) {
    const float4* at = reinterpret_cast<const float4*>(place(i)) + row * (width / 4) + 2 * piece;
    const float4 a = at[0], b = at[1];
    MtEight e = {{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
    return e;
  };
  auto mine = [&](int i, bool values) { return place(i) + (values ? MT_C * MT_C * 4 : MT_C * MT_M * 4) + tid * 16; };

  MtUnit c = {};                                 // the tile in work
  OnePlace copies[2];                            // (of thread 0)
  auto gave_up = [&]() { return *(volatile int*)&sh.abort != 0; };
  // step `i` of all, a tile's `step` (all have read the step before last; rows beyond the last repeat it: q's
  // results are not stored, values' weights are zero)
  auto fetch = [&](const MtUnit& c, int step, int i) {
    const size_t head = (size_t)c.chunk * p.H + c.h;
    uint8_t* to = place(i);
    uint64_t* got = sh.got + (i & 1);
    if (step < steps) {
      if (tid == 0) {
        copies[i & 1].fill(gave_up(), [&]() {
          mbar_expect_tx(got, MT_C * MT_M * 4 + MT_C * 4);
          bf_bulk_load(n_s[i & 1], Un + head * p.dk + step * MT_C, MT_C * 4, got);
          bf_bulk_load(to, U + head * p.dk * p.dv + (size_t)c.m0 * p.dk + step * MT_C * MT_M, MT_C * MT_M * 4, got);
        });
      }
      mt_fetch(mine(i, false), proj + (size_t)(c.t0 + min(tr, c.n - 1)) * p.qk_stride + p.q_off +
                                   (size_t)c.h * p.dk + step * MT_C + 8 * tq);
    } else {
      if (tid == 0) {
        copies[i & 1].fill(gave_up(), [&]() {
          mbar_expect_tx(got, MT_C * MT_C * 4);
          bf_bulk_load(to, qkm + head * MT_C * MT_C, MT_C * MT_C * 4, got);
        });
      }
      const mt_bf16* v = proj + (size_t)c.t0 * p.v_stride + p.v_off + (size_t)c.h * p.dv + c.m0 + 8 * mq;
      uint8_t* at = mine(i, true);
      mt_fetch(at, v + (size_t)min(mr, c.n - 1) * p.v_stride);
      mt_fetch(at + 16 * MT_WORK, v + (size_t)min(mr + 32, c.n - 1) * p.v_stride);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // q . k with its weight: row t sees the chunk's tokens up to itself
  auto weighted = [&](const MtTable& tb, int i) {
    const int t = tr, s = 8 * tq, last = t < c.n ? t : -1, b = s >> 4;
    MtEight e = {};
    if (s > last) return e;
    e = eight(i, t, MT_C, tq);
    if (b < t >> 4) {
      const float2 r = tb.row[b][t];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 k = tb.col[s + j];
        const float hi = r.x * k.x;
        e.v[j] = cs_times(e.v[j], make_float2(hi, fmaf(r.x, k.x, -hi) + fmaf(r.x, k.y, r.y * k.x)));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) e.v[j] = s + j <= last ? cs_times(e.v[j], tb.near[t][(s + j) & 15]) : 0.f;
    }
    return e;
  };
  float den = 0.f;                               // n_t . q_t, this thread's share of row tr
  auto convert = [&](MtTable& tb, int step, int i) {
    uint8_t* tm = ring + (i & 1) * MT_OUT_STAGE + m_spot;
    uint8_t* tt = ring + (i & 1) * MT_OUT_STAGE + (step < steps ? 3 : 1) * MT_TILE + t_spot;
    float2 left = make_float2(0.f, 0.f);
    // (two steps are asked for; of tiles of two steps, whose next is known late, both or none)
    if (steps > 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    mbar_wait(sh.got + (i & 1), (i >> 1) & 1, &sh.abort);
    auto raw = [&](int x) {
      return *reinterpret_cast<const uint4*>(mine(i, step == steps) + x * 16 * MT_WORK);
    };
    if (step < steps) {
#pragma unroll
      for (int x = 0; x < 2; ++x) mt_put(tm + x * 4096, MT_TILE, eight(i, mr + 32 * x, MT_M, mq), left);
      const uint4 qv = raw(0);
      *reinterpret_cast<uint4*>(tt) = qv;
      {
        const MtEight f = mt_bf16s(qv);
        const float4 a = *reinterpret_cast<const float4*>(n_s[i & 1] + 8 * tq);
        const float4 b = *reinterpret_cast<const float4*>(n_s[i & 1] + 8 * tq + 4);
        den += ((f.v[0] * a.x + f.v[1] * a.y) + (f.v[2] * a.z + f.v[3] * a.w)) +
               ((f.v[4] * b.x + f.v[5] * b.y) + (f.v[6] * b.z + f.v[7] * b.w));
      }
      if (mt_bad(left) || mt_bad(qv)) {
#pragma unroll 1
        for (int x = 0; x < 2; ++x) {
          MtEight e = eight(i, mr + 32 * x, MT_M, mq);
          const int bad = mt_clean(e, MT_NO_TERMS_UP);
          for (int j = 0; j < 8; ++j)
            if (bad >> j & 1) tb.odd_m[8 * mq + j] = 0;
          mt_put(tm + x * 4096, MT_TILE, e, left);
        }
        MtEight f = mt_bf16s(qv);
        if (mt_clean(f, MT_NO_TERMS)) tb.odd_t[tr] = 1;
        *reinterpret_cast<uint4*>(tt) = mt_pack(f);
        tb.odd = 1;
      }
      return;
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      uint4 v = raw(x);
      if (mt_bad(v)) {
        MtEight f = mt_bf16s(v);
        const int bad = mt_clean(f, MT_NO_TERMS);
        for (int j = 0; j < 8; ++j)
          if (bad >> j & 1) atomicMin(tb.odd_m + 8 * mq + j, mr + 32 * x);
        v = mt_pack(f);
        tb.odd = 1;
      }
      *reinterpret_cast<uint4*>(tm + x * 4096) = v;
    }
    MtEight w = weighted(tb, i);
    // n_t . q_t: the state's share with the token's weight, and the row's sum
    den = cs_times(den, tb.at[tr]);
    if (!(fabsf(den) < INFINITY) && tr < c.n) {  // (the weight on q: it may keep the products finite)
      const mt_bf16* q = proj + (size_t)(c.t0 + tr) * p.qk_stride + p.q_off + (size_t)c.h * p.dk + 8 * tq;
      const float* n = Un + ((size_t)c.chunk * p.H + c.h) * p.dk + 8 * tq;
      den = 0.f;
#pragma unroll 1
      for (int k = 0; k < p.dk; k += MT_C)
#pragma unroll 1
        for (int j = k; j < k + 8; ++j) den = fmaf(cs_times(bf_ld(q + j), tb.at[tr]), n[j], den);
    }
    den +=
          (((w.v[0] + w.v[1]) + (w.v[2] + w.v[3])) + ((w.v[4] + w.v[5]) + (w.v[6] + w.v[7])));
    mt_put(tt, MT_TOK, w, left);
    if (mt_bad(left)) {
      mt_clean(w, MT_NO_TERMS_UP);
      tb.odd_t[tr] = 1;
      tb.odd = 1;
      mt_put(tt, MT_TOK, w, left);
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    if (tq == 0) tb.den[tr] = tr < c.n ? fmaxf(fabsf(den), E[(size_t)c.h * p.T + c.t0 + tr]) + 1e-6f : 1.f;
  };
  unsigned long long sum[8];                     // (times SPLIT_UP)
  auto finish = [&](const MtTable& tb, int step, int i) {
    mt_done(sh, i);
#pragma unroll
    for (int j0 = 0; j0 < 8; j0 += 4) {
      unsigned long long u[4];
      mt_take(from + (uint32_t)((i & 1) * 3 * MT_C + 2 * j0), u);
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[j0 + j] = step ? cs_add2(sum[j0 + j], u[j]) : u[j];
    }
    if (step == steps - 1) {                     // times the tokens' weights
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float a, b;
        cs_unpair(sum[j], a, b);
        sum[j] = cs_pair(cs_times(a, tb.at[group * 16 + 2 * j]), cs_times(b, tb.at[group * 16 + 2 * j + 1]));
      }
    }
    if (step < steps) return;
    const MtUnit& x = tb.unit;
    const size_t row = (size_t)p.H * p.dv;
    float* dst = o_raw + (size_t)(x.t0 + group * 16) * row + (size_t)x.h * p.dv + x.m0 + m;
    const int n = x.n - group * 16;
    unsigned lost = 0;                           // tokens whose sum is not finite
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float a, b;
      cs_unpair(sum[j], a, b);
      lost |= (fabsf(a) < INFINITY ? 0u : 1u << 2 * j) | (fabsf(b) < INFINITY ? 0u : 2u << 2 * j);
      if (2 * j < n) dst[0] = a * SPLIT_DOWN / tb.den[group * 16 + 2 * j];
      if (2 * j + 1 < n) dst[row] = b * SPLIT_DOWN / tb.den[group * 16 + 2 * j + 1];
      dst += 2 * row;
    }
    if (!tb.odd && !lost) return;
    // (in cs_out's order: runs of sixteen, the weight on q)
#pragma unroll 1
    for (int t = group * 16; t < min(group * 16 + 16, x.n); ++t) {
      if (!tb.odd_t[t] && tb.odd_m[m] > t && !(lost >> (t & 15) & 1)) continue;
      const mt_bf16* q = proj + (size_t)(x.t0 + t) * p.qk_stride + p.q_off + (size_t)x.h * p.dk;
      const mt_bf16* v = proj + (size_t)x.t0 * p.v_stride + p.v_off + (size_t)x.h * p.dv + x.m0 + m;
      const float* P = qkm + (((size_t)x.chunk * p.H + x.h) * MT_C + t) * MT_C;
      const float* S = U + ((size_t)x.chunk * p.H + x.h) * p.dk * p.dv + (size_t)x.m0 * p.dk + m;
      float o = 0.f;
#pragma unroll 1
      for (int k0 = 0; k0 < p.dk; k0 += 16) {
        float run = 0.f;
#pragma unroll 1
        for (int k = k0; k < k0 + 16; ++k)
          run = fmaf(cs_times(bf_ld(q + k), tb.at[t]), S[(size_t)k * MT_M], run);
        o += run;
      }
#pragma unroll 1
      for (int y0 = 0; y0 <= t; y0 += 16) {
        float run = 0.f;
#pragma unroll 1
        for (int y = y0; y <= min(t, y0 + 15); ++y)
          run = fmaf(cs_times(P[y], cs_exp(tb.g[t] - tb.h[y])), bf_ld(v + (size_t)y * p.v_stride), run);
        o += run;
      }
      o_raw[(size_t)(x.t0 + t) * row + (size_t)x.h * p.dv + x.m0 + m] = o / tb.den[t];
    }
  };

  int i = 0, tab = 0;
  double gn = 0.0, hn = 0.0, before = 0.0;       // of the next tile's token tid
  auto sums = [&](const MtUnit& c) {             // a tile's token tid
    if (c.b < 0 || tid >= MT_C) return;
    const size_t t = (size_t)c.h * p.T + c.t0;
    before = c.index ? G[t - 1] : g0[(size_t)c.b * p.H + c.h];
    gn = G[t + min(tid, c.n - 1)];
    hn = Hs[t + min(tid, c.n - 1)];
  };
  __syncthreads();                               // (the first tile is found)
  c = next_s;
  sums(c);
  if (c.b >= 0) {
    fetch(c, 0, 0);
    fetch(c, 1, 1);
  }
  while (c.b >= 0) {
    // ---- the tile's tables (the tile before last, whose place they take, is finished)
    MtTable& tb = table[tab];
    if (tid < MT_C) {
      const double x = tid < c.n ? gn : 0.0;
      tb.g[tid] = x;
      tb.h[tid] = tid < c.n ? hn : 0.0;
      float2 w = make_float2(0.f, 0.f);
      if (tid < c.n) {
        w = cs_exp(x - before);
        // (times q_scale: its products' roundings are part of what is left)
        const float f = w.x * p.q_scale;
        w = make_float2(f, fmaf(w.x, p.q_scale, -f) + w.y * p.q_scale);
        if (!(fabsf(f) < INFINITY)) w.y = 0.f;
      }
      tb.at[tid] = w;
      tb.odd_t[tid] = 0;
      if (tid == 0) {
        tb.odd = 0;
        tb.unit = c;
      }
    } else if (tid < MT_C + MT_M) {
      tb.odd_m[tid - MT_C] = MT_C;
    }
    den = 0.f;
    __syncthreads();
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int t = (tid >> 4) + 32 * x, s = (t & 48) + (tid & 15);
      if (s <= t && t < c.n) tb.near[t][tid & 15] = cs_exp(tb.g[t] - tb.h[s]);
    }
    if (tid < 256) {
      const int t = tid & 63, b = tid >> 6;      // b 3: the columns' factors
      if (b < 3) {
        if (t >= 16 * b + 16 && t < c.n) tb.row[b][t] = cs_exp(tb.g[t] - tb.g[16 * b + 15]);
      } else if (t < 48 && (t | 15) < c.n) {
        tb.col[t] = cs_exp(tb.g[t | 15] - tb.h[t]);
      }
    }
    MtUnit after = {};                           // the tile behind it: known from its second step on
    for (int step = 0; step <= steps; ++step, ++i) {
      convert(tb, step, i);
      mt_stored();
      if (step == 1) after = next_s;
      if (step + 2 <= steps) {
        fetch(c, step + 2, i + 2);
      } else if (step > 0 && after.b >= 0) {
        if (steps == 1) fetch(after, 0, i + 1);
        fetch(after, step + 1 - steps, i + 2);
      } else {
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      if (step == steps) sums(after);
      if (step) finish(tb, step - 1, i - 1);
      else if (i) finish(table[tab ^ 1], steps, i - 1);
    }
    tab ^= 1;
    c = after;
  }
  if (i) finish(table[tab ^ 1], steps, i - 1);
  if (tid == 0 && gave_up())                     // (a copy that this thread did not see land)
    for (int x = 0; x < 2; ++x) copies[x].drain([&](int, unsigned parity) { mbar_drain_one(sh.got + x, parity); });
  mt_end(sh, tmem, err);
}

// Chunks of 64 (tokens), keys in whole steps, values in whole tiles, rows on 16-byte boundaries.  And CTAs
// for the chip: mt_state goes from chunk to chunk with one for 64 x 128 elements of a state, where cs_state
// has one for every chunk, too.  On the tensor cores / multiply-adds, 2,048 tokens: 48 CTAs 175 / 194 and
// 185 / 202 us, 32 CTAs 161 / 149, 165 / 153 and 192 / 200, 16 CTAs 149 / 116 and 157 / 122, one 124 / 67;
// 8,192 tokens, 48: 576 / 650, 16: 470 / 302.  Up to five chunks the former are no slower whatever the CTAs
// (200 tokens: 52 to 77 us against 52 to 89).  `min_ctas`: 40.  max_q: the step's longest portion (0: not
// known); requests of up to n_min tokens have no chunks.
static bool mt_takes(const CsIn& p, const void* proj, int chunks, int max_q, int min_ctas) {
  const int longs = max_q > 0 ? 1 + (p.T > max_q ? p.T - max_q : 0) / (p.n_min + 1) : p.T / (p.n_min + 1);
  const long long ctas = (long long)(p.dk / MT_C) * (p.dv / MT_M) * p.H * (p.B < longs ? p.B : longs);
  return (ctas >= min_ctas || chunks <= 5) &&
         (long long)chunks * p.H * (p.dv / MT_M) < 0x7fffffff && p.C == MT_C && p.dk % MT_C == 0 && p.dk <= MT_WORK && p.dv % MT_M == 0 && p.qk_stride % 8 == 0 &&
         p.q_off % 8 == 0 && p.k_off % 8 == 0 && p.v_off % 8 == 0 && ((uintptr_t)proj & 15) == 0;
}
static int mt_launch(const mt_bf16* proj, const CsIn& p, int chunks, const int* q_start, float* state,
                     long long slot_stride, int state_size, const int* state_slots, int n_slots, const double* G,
                     const double* Hs, const double* g0, const float2* Wl, const float* E, const float* qkm,
                     float* U, float* Un, float* o_raw, int* err, cudaStream_t stream) {
  static bool configured_on[BF_MAX_DEVICES];
  bool& configured = configured_on[bf_current_device()];
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(mt_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         MT_STATE_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mt_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_OUT_SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  mt_state_kernel<<<dim3(p.dv / MT_M * (p.dk / MT_C), p.H, p.B), MT_THREADS, MT_STATE_SMEM, stream>>>(
      proj, p, q_start, state, slot_stride, state_size, state_slots, n_slots, G, g0, Wl, U, Un, err);
  const long long units = (long long)chunks * p.H * (p.dv / MT_M);
  mt_out_kernel<<<(unsigned)(units < 148 ? units : 148), MT_THREADS, MT_OUT_SMEM, stream>>>(
      proj, p, chunks, q_start, state_slots, n_slots, G, Hs, g0, E, qkm, U, Un, o_raw, err);
  return bf_launch_status();
}
