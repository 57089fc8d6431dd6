// The products of the chunks' float recurrences (chunk_scan.cu: linear scan, delta rule) on the 5th-generation
// tensor cores.  Every operand is a float in three bfloat16 terms (split_utils.cuh), a product of two floats
// the six products of terms that matter.
//
//   cs_qk      leaves q and k in terms, once for all heads that share them, in the tiles that the products read
//   ct_weights q . k with the weights of a head's tokens
//   ct_state   what cs_state and cs_prefix compute: a CTA keeps 128 key x 32 value sizes of a head's state in
//              registers and goes from chunk to chunk; the states between the chunks are written once
//   dt_walk    what ds_walk computes, the delta rule's chain
//   ct_out     what cs_out computes: 128 value sizes (of one head, or of two heads of 64) x 64 tokens a tile,
//              a CTA an SM goes from tile to tile
//
// ct_state and ct_out have a warp that asks for the terms' tiles, warps that weight the other operand, take it apart
// and store its terms, two warps that issue the products in turn and warps that take the sums out of tensor memory and
// add; each goes ahead as far as rings of two to four places let it.  (One set of warps that did all of it in
// turn spent three quarters of its time waiting for its own copies and sums.)  dt_walk's two products a chunk wait
// for one another, so the warps that keep the state do both there.
//
// A step has 64 terms.  Products of a leading term with all three of the other side go out as one instruction
// of three times the columns, so a step's rows are read from shared memory three times and not six:
//
//   rows' hi x [hi | mid | lo], rows' mid x [hi | mid], rows' lo x [hi]
//
// The tensor core's sums cut where arithmetic rounds, so the leading terms' products are summed 32 terms at a
// time, apart from the smaller ones', and the sums are added in rounded float.  Floats are multiplied by 2^24
// before they are taken apart, so that their terms hold them whatever their size, and the sums by 2^-48.
// Operands that have no terms (infinities, NaN, floats from 2^104 on) are zero in the products, and what they
// reach is computed by multiply-adds in cs_state's and cs_out's order; so are sums that are not finite.
//
// 2,000 tokens of 64 heads of 128 x 64 over 8: ct_state 36 us (cs_state and cs_prefix 87), ct_weights 15, ct_out 58
// (cs_out 100); 1,300 and 812 tokens of 8 heads of 128 x 256: 25 (47), 5, 30 (58); the delta rule's 1,111 and 694 of
// 16 heads of 128: dt_walk 59 (ds_walk 108), ct_out 31 (cs_out 53), ds_prep 39 (47).  What bounds ct_out is the rate
// at which its warps get instructions (0.45 a cycle and scheduler): its time changes by 0 to 3 us without its
// stores, with loads that always hit, with half of the products or without taking the operands apart.  ct_state and
// dt_walk are bound by their chains: some 1,460 (25 of its 35 us at 32 chunks; the rest is its start and end) and
// 4,600 cycles a chunk.  (With a row of the state a thread, half as many warps, they were 39 and 70 us.)
// Relative errors against 64 bits (outputs, states), these / multiply-adds, e-7: decays of 0.98 to 1 0.78 0.66 / 1.32
// 1.28, a state space layer's 0.55 0.46 / 0.68 0.59, spread over 0 to 1 0.51 0.43 / 0.54 0.42, a tenth of those zero
// 0.50 0.42 / 0.51 0.37; the delta rule's 0.91 0.85 / 1.61 1.80, 0.66 0.59 / 0.77 0.68, 0.60 0.56 / 0.66 0.50, 0.58
// 0.52 / 0.64 0.46.  Where a state is made up of a few tokens, as with the last two, it is up to 0.06e-7 further
// off (half a unit in the last place is 0.6e-7): its last terms' sum is cut, one more loss of the size of a rounding.
// More or less than ct_take's 2^-25 is no way out (delta, spread and zeros: none 0.66 0.55, half of it 0.59 0.51,
// three quarters 0.57 0.51), nor are the products of terms that are left out (0.557 0.514, and 5 us more of 139) or
// both roundings of the last additions kept (no change).
//
// Included by chunk_scan.cu behind mlstm_tensor.cuh.
#pragma once

#define CT_C 64                       // tokens of a chunk, and terms of a step
#define CT_TERM CS_TERMS_TERM         // a term of a tile: 64 rows (tokens) of 64 numbers
#define CT_TILE CS_TERMS_TILE         // 64 tokens x 64 sizes of q or k
constexpr float CT_DOWN = SPLIT_DOWN * SPLIT_DOWN;
constexpr float CT_CUT = 1.f / 33554432.f;               // 2^-25

__device__ __forceinline__ unsigned long long ct_mul2(unsigned long long x, unsigned long long y) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ unsigned long long ct_mul2(unsigned long long x, float f) {
  return ct_mul2(x, cs_pair(f, f));
}

// Rows' terms MN-major in blocks of 64 (`lbo` bytes apart; a term `term_a` bytes behind the one before) times
// columns' terms K-major, N of them a term behind one another: sums of the leading products' first 32 terms
// at `d`, of the others at d + N and d + 2 N, of the leading ones' last 32 at d + 3 N.
template <int N>
__device__ __forceinline__ void ct_products(uint32_t d, uint32_t a, uint32_t term_a, uint32_t lbo, uint32_t b) {
  constexpr uint32_t base = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((uint32_t)(128 >> 4) << 24);
  constexpr uint32_t one = base | ((uint32_t)(N >> 3) << 17), two = base | ((uint32_t)(2 * N >> 3) << 17),
                     three = base | ((uint32_t)(3 * N >> 3) << 17);
  const uint64_t hi = umma_desc_mn_sw128(a, lbo), mid = umma_desc_mn_sw128(a + term_a, lbo),
                 lo = umma_desc_mn_sw128(a + 2 * term_a, lbo), bh = umma_desc_k_sw128(b),
                 bm = umma_desc_k_sw128(b + N * 128);
#pragma unroll
  for (int k = 0; k < 4; ++k) {                // (16 terms further: 16 rows; 32 bytes)
    const uint64_t ka = (uint64_t)(k * 16 * 128 >> 4), kb = (uint64_t)(k * 32 >> 4);
    if (k < 2) {
      umma_bf16(d, hi + ka, bh + kb, three, k > 0);
    } else {
      umma_bf16(d + 3 * N, hi + ka, bh + kb, one, k > 2);
      umma_bf16(d + N, hi + ka, bm + kb, two, 1);
    }
    umma_bf16(d + N, mid + ka, bh + kb, two, 1);
    umma_bf16(d + 2 * N, lo + ka, bh + kb, one, 1);
  }
}

// Eight columns of such a step's four places: the sums of the leading products' 32 terms that come last (`second`:
// the second 32), and of all others.  Where decays are fast the last terms make up the result, so they are added
// last; and their sum, which the tensor core cuts, is half a unit too small on average: 2^-25 of it is added to the
// others (less than half a unit, so that a sum that is exact stays so).
template <int N>
__device__ __forceinline__ void ct_take(uint32_t at, bool second, unsigned long long (&last)[4],
                                        unsigned long long (&rest)[4]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%33];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%34];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%35];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(second ? at : at + 3 * N), "r"(at + N), "r"(at + 2 * N), "r"(second ? at + 3 * N : at)
      : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    unsigned long long x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      x[k] = cs_pair(__uint_as_float(r[8 * k + 2 * i]), __uint_as_float(r[8 * k + 2 * i + 1]));
    last[i] = x[3];
    rest[i] = cs_add2(x[0], cs_fma2(x[3], cs_pair(CT_CUT, CT_CUT), cs_add2(x[1], x[2])));
  }
}

// mbar_wait with the hint that a thread may sleep for some microseconds: warps that wait took issue slots from
// those that work
__device__ __forceinline__ bool ct_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool ct_wait(uint64_t* bar, uint32_t parity, volatile int* abort) {
  if (ct_try(bar, parity)) return true;
  const long long t0 = clock64();
  while (!ct_try(bar, parity)) {
    if (*abort) return false;
    if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
      *abort = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool ct_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort) {
  const bool ok = ct_wait(bar, parity, abort);
  return __all_sync(0xffffffffu, ok);
}

// What other threads stored ahead of a barrier that this one has passed is there for the products: a proxy fence
// anywhere on the way from a write to the other proxy's read orders them.  (By the warp that issues the products and
// not by those that store: there it waits for a thread's loads, too, and theirs are for the step behind; ct_out 61 us
// so, 58 here.)
__device__ __forceinline__ void ct_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void ct_arrive(uint64_t* bar) {      // by a warp: its writes are done
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

struct CtShared {
  uint64_t full[3], free[3];          // tiles of terms (by the copy; by the products' commit)
  uint64_t put[2], done[2], taken[2]; // the other operand's places, the sums' places
  uint64_t w_put[2], w_free[2];       // ct_out: the weighted q . k's places
  uint64_t a_free[2], drain;          // ct_out: the rows' places
  uint32_t tmem;
  int abort;
};
template <int COLS>
__device__ __forceinline__ uint32_t ct_begin(CtShared& s, int warp, int alloc_warp) {
  if (warp == alloc_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s.tmem)),
                 "r"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return s.tmem;
}
// (products are issued by warps `mma_warp` and the one behind it: `drain` takes two arrivals)
template <int COLS>
__device__ __forceinline__ void ct_end(CtShared& s, uint32_t tmem, int warp, int mma_warp, int* err) {
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  if (*(volatile int*)&s.abort) {                        // (a wait gave up)
    if (threadIdx.x == 0) atomicOr(err, BF_ERR_WAIT);
    if (warp == mma_warp || warp == mma_warp + 1) {      // products still in flight
      umma_commit(&s.drain);
      const long long t0 = clock64();
      while (!mbar_try_wait(&s.drain, 0) && clock64() - t0 < WAIT_LIMIT_CYCLES / 16) {
      }
    }
    __syncwarp();
    __syncthreads();
  }
  if (warp == mma_warp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS)
                 : "memory");
  }
}

// ------------------------------------------------------------------------------ ct_weights
// What ct_out needs of a chunk and head, from G and H (ct_weights)
struct CtHead {
  float at[2][CT_C];                                     // the tokens' weights of the state before, times q_scale;
                                                         // what is left of them
  float P[CT_C][CT_C];                                   // exp(G_t - H_s) (q_t . k_s), in the blocks of 16 x 16 up
};                                                       // to the diagonal
// and on the way, floats and what is left of them
struct CtWeights {
  double g[CT_C], h[CT_C];
  float near[2][CT_C][16];                               // exp(G_t - H_s) inside a block of 16
  float row[2][3][CT_C];                                 // exp(G_t - G of block b's end)
  float col[2][48];                                      // exp(that - H_s)
};

// By a block of 256 threads; g, hs: G and H of the chunk's n tokens, before: G of the token ahead of them, at: CtHead's
// or null.  Where s lies in an earlier block of 16 tokens than t, exp(G_t - H_s) is two factors by the block's last G,
// each a float and what is left of it: some 700 exponentials and not 2,080.  Returns true where a factor is above 1,
// as decays above 1 make it: the other one may then lie below the normal floats while the product does not, and
// whoever asks takes the exponential itself.
__device__ __forceinline__ bool ct_factors(const double* g, const double* hs, double before, int n, float q_scale,
                                           CtWeights& w, float (*__restrict__ at)[CT_C]) {
  const int tid = threadIdx.x;
  if (tid < 2 * CT_C) (tid < CT_C ? w.g : w.h)[tid % CT_C] = tid % CT_C < n ? (tid < CT_C ? g : hs)[tid % CT_C] : 0.0;
  __syncthreads();
  // (rows q and 15 - q of a block have 17 columns up to the diagonal; 48, 32 and 16 rows behind blocks 0, 1, 2.
  // A thread's three exponentials side by side: ds_prep 2 us less)
  double d[3];
  float *to[3], *left[3];
  bool scaled = false, above = false;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const int i = tid + 256 * x;
    int gi = CT_C;
    float *dst = nullptr, *rest = nullptr;
    double from = 0.0;
    if (i < 32 * 17) {
      const int pair = i / 17, c = i - pair * 17, q = pair & 7;
      const int r = c <= q ? q : 15 - q, col = c <= q ? c : c - q - 1;
      gi = (pair >> 3) * 16 + r;
      from = w.h[(pair >> 3) * 16 + col];
      dst = &w.near[0][gi][col];
      rest = &w.near[1][gi][col];
    } else if (i < 32 * 17 + 96) {
      const int c = i - 32 * 17, bl = c < 48 ? 0 : c < 80 ? 1 : 2;
      gi = c - (bl == 0 ? 0 : bl == 1 ? 48 : 80) + 16 * bl + 16;
      from = w.g[16 * bl + 15];
      dst = &w.row[0][bl][gi];
      rest = &w.row[1][bl][gi];
    } else if (i < 32 * 17 + 144) {
      const int c = i - 32 * 17 - 96;
      gi = c | 15;
      from = w.h[c];
      dst = &w.col[0][c];
      rest = &w.col[1][c];
    } else if (at && i < 32 * 17 + 144 + CT_C) {
      gi = i - 32 * 17 - 144;
      from = before;
      dst = &at[0][gi];
      rest = &at[1][gi];
      scaled = x == 2;
    }
    d[x] = gi < n ? w.g[gi] - from : -INFINITY;          // (0 for rows that are not there)
    above |= i >= 32 * 17 && i < 32 * 17 + 144 && d[x] > 0.0;
    to[x] = dst;
    left[x] = rest;
  }
  float2 e[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) e[x] = cs_exp<true>(d[x]);
  if (scaled) {                                          // (the product's roundings are part of what is left)
    const float f = e[2].x * q_scale;
    e[2] = make_float2(f, fmaf(e[2].x, q_scale, -f) + e[2].y * q_scale);
    if (!(fabsf(f) < INFINITY)) e[2].y = 0.f;
  }
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    if (!to[x]) continue;
    *to[x] = e[x].x;
    *left[x] = e[x].y;
  }
  return __syncthreads_or(above);
}
// the weights of a row's octet as exponentials of their own
__device__ __noinline__ void ct_weights_again(const CtWeights& w, int t, int s, int n, const float* __restrict__ pm,
                                              CtHead* __restrict__ to) {
#pragma unroll 1
  for (int c = s; c < s + 8; ++c)
    to->P[t][c] = t < n && c <= t ? cs_times(pm[t * CT_C + c], cs_exp(w.g[t] - w.h[c])) : 0.f;
}
// pm: the chunk's q . k, above: ct_factors'
__device__ __forceinline__ void ct_weights(const CtWeights& w, int n, bool above, const float* __restrict__ pm,
                                           CtHead* __restrict__ to) {
  const int tid = threadIdx.x;
  // row tid / 4, octets tid % 4 and four further
  const int t = tid >> 2;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int s = 8 * ((tid & 3) + 4 * x), cb = s >> 4;
    if (cb > t >> 4) continue;
    const bool own = cb == t >> 4;
    if (above && !own) {
      ct_weights_again(w, t, s, n, pm, to);
      continue;
    }
    const float rx = own ? 0.f : w.row[0][cb][t], ry = own ? 0.f : w.row[1][cb][t];
    const int last = t < n ? t - s : -1;
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      float4 v = *reinterpret_cast<const float4*>(pm + t * CT_C + s + j);
      float4 hi = *reinterpret_cast<const float4*>(own ? &w.near[0][t][(s & 15) + j] : &w.col[0][s + j]);
      float4 lo = *reinterpret_cast<const float4*>(own ? &w.near[1][t][(s & 15) + j] : &w.col[1][s + j]);
      auto one = [&](float a, float cx, float cy, int at) {
        float2 f = make_float2(cx, cy);
        if (!own) {                                      // (r + what is left) (c + what is left)
          f.x = rx * cx;
          f.y = fmaf(rx, cx, -f.x) + fmaf(rx, cy, ry * cx);
        }
        return j + at <= last ? cs_times(a, f) : 0.f;
      };
      *reinterpret_cast<float4*>(&to->P[t][s + j]) =
          make_float4(one(v.x, hi.x, lo.x, 0), one(v.y, hi.y, lo.y, 1), one(v.z, hi.z, lo.z, 2),
                      one(v.w, hi.w, lo.w, 3));
    }
  }
}
// grid (chunks, H)
__global__ void __launch_bounds__(256) ct_weights_kernel(CsIn p, const int* __restrict__ q_start,
                                                         const double* __restrict__ G,
                                                         const double* __restrict__ Hs,
                                                         const double* __restrict__ g0,
                                                         const float* __restrict__ qkm, CtHead* __restrict__ W) {
  __shared__ __align__(16) CtWeights w;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, blockIdx.x, -1);
  if (c.b < 0) return;
  const int at = c.index * CT_C, h = blockIdx.y, hq = h / (p.H / p.QH);
  const double* g = G + (size_t)h * p.T + c.t0 + at;
  const int n = min(CT_C, c.n - at);
  CtHead* to = W + (size_t)blockIdx.x * p.H + h;
  const bool above =
      ct_factors(g, Hs + (g - G), c.index ? g[-1] : g0[(size_t)c.b * p.H + h], n, p.q_scale, w, to->at);
  ct_weights(w, n, above, qkm + ((size_t)blockIdx.x * p.QH + hq) * CT_C * CT_C, to);
}

// -------------------------------------------------------------------------------- ct_state
// grid (tiles of 128 key x 32 value sizes of a head's state, H, B).  The products' rows are key sizes: k's
// tiles come as they are, and what a CTA takes apart are its own 32 value sizes of a chunk.  The state lies as
// [dv][dk]; between the chunks (U): [dv / 32][dk][32], a row's pieces of sixteen bytes p at p ^ (row % 8),
// so that a CTA's elements are one block, which leaves through shared memory in one copy.
#define CT_SV 32                                         // value sizes of a CTA
#define CT_S_RING 3                                      // places for k's tiles
#define CT_S_KEYS (2 * CT_TILE)                          // 64 tokens x 128 sizes
#define CT_S_VALS (3 * CT_SV * 128)                      // the values' terms
#define CT_S_RAW (CT_C * CT_SV * 4)                      // and as they come
#define CT_S_SMEM (1024 + CT_S_RING * CT_S_KEYS + 2 * CT_S_VALS + 128 * CT_SV * 4 + 4 * (CT_S_RAW + CT_C * 8))
#define CT_S_THREADS 480             // eight warps that add, four that convert, one that copies, two for products
#define CT_S_COLS 256                                    // tensor memory: two places of 4 x 32 columns

// the chunk's share of 16 elements of the state by multiply-adds, as cs_state sums it
__device__ __noinline__ void ct_state_again(const float* __restrict__ k, long long k_stride,
                                            const float* __restrict__ v, long long v_stride,
                                            const float2* __restrict__ wl, int n, float* u) {
#pragma unroll 1
  for (int j0 = 0; j0 < CT_SV / 2; j0 += 8) {
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int s = 0; s < n; ++s) {
      const float x = k[(size_t)s * k_stride];
      const float2 w = wl[s];
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = fmaf(cs_times(v[(size_t)s * v_stride + j0 + j], w), x, a[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) u[j0 + j] = a[j];
  }
}

__global__ void __launch_bounds__(CT_S_THREADS, 1) ct_state_kernel(
    const float* __restrict__ qk, const float* __restrict__ vsrc, CsIn p, const int* __restrict__ q_start,
    float* __restrict__ state, long long slot_stride, const int* __restrict__ state_slots, int n_slots,
    const double* __restrict__ G, const float2* __restrict__ Wl, const uint8_t* __restrict__ Xk,
    const unsigned long long* __restrict__ odd_rows, float* __restrict__ U, int* __restrict__ err) {
  extern __shared__ __align__(16) uint8_t ct_raw[];
  __shared__ CtShared sh;
  __shared__ int odd_v[4][CT_SV];                        // (of chunk % 4) chunk + 1: the column has no terms
  uint8_t* keys = ct_raw + ((1024u - (smem_u32(ct_raw) & 1023u)) & 1023u);
  uint8_t* vals = keys + CT_S_RING * CT_S_KEYS;
  float* kept = reinterpret_cast<float*>(vals + 2 * CT_S_VALS);          // [128][32]
  uint8_t* raw = reinterpret_cast<uint8_t*>(kept + 128 * CT_SV);         // [4][4 warps][16 tokens][32]
  float2* raw_w = reinterpret_cast<float2*>(raw + 4 * CT_S_RAW);         // [4][4 warps][16]
  const int h = blockIdx.y, b = blockIdx.z;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, 0, b);
  if (c.n <= p.n_min) return;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= n_slots) {
    if (threadIdx.x == 0) atomicOr(err, BF_ERR_SLOT);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_k = p.dk / 128;
  const int k0 = (int)blockIdx.x % tiles_k * 128, v0 = (int)blockIdx.x / tiles_k * CT_SV;
  const int hq = h / (p.H / p.QH);
  const int chunks = (c.n + CT_C - 1) / CT_C;
  const float* vp = vsrc + (size_t)c.t0 * p.v_stride + p.v_off + (size_t)h * p.dv + v0;
  const float2* wl = Wl + (size_t)h * p.T + c.t0;
  if (tid == 0) {
    for (int i = 0; i < CT_S_RING; ++i) {
      mbar_init(sh.full + i, 1);
      mbar_init(sh.free + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(sh.put + i, 4);
      mbar_init(sh.done + i, 1);
      mbar_init(sh.taken + i, 8);
    }
    mbar_init(&sh.drain, 2);
    sh.abort = 0;
  }
  if (tid < 4 * CT_SV) odd_v[tid / CT_SV][tid % CT_SV] = 0;
  const uint32_t tmem = ct_begin<CT_S_COLS>(sh, warp, 13);

  if (warp == 12) {                                      // ---- k's tiles
    if (lane == 0) {
      int place = 0;
      uint32_t phase = 0;
      const uint8_t* X = Xk + (((size_t)c.first * p.QH + hq) * (p.dk / 64) + k0 / 64) * CT_TILE;
      const size_t step = (size_t)p.QH * (p.dk / 64) * CT_TILE;
      for (int i = 0; i < chunks; ++i) {
        if (i >= CT_S_RING && !ct_wait(sh.free + place, phase ^ 1u, &sh.abort)) break;
        mbar_expect_tx(sh.full + place, CT_S_KEYS);
        bf_bulk_load(keys + place * CT_S_KEYS, X + i * step, CT_S_KEYS, sh.full + place);
        if (++place == CT_S_RING) place = 0, phase ^= 1u;
      }
      if (*(volatile int*)&sh.abort) mbar_drain(sh.full, CT_S_RING, place, phase);
    }
    __syncwarp();
  } else if (warp >= 13) {                               // ---- products: chunks in turn
    for (int i = warp - 13; i < chunks; i += 2) {
      const int place = i % CT_S_RING;
      ct_wait_warp(sh.full + place, (i / CT_S_RING) & 1, &sh.abort);
      ct_wait_warp(sh.put + (i & 1), (i >> 1) & 1, &sh.abort);
      if (i >= 2) ct_wait_warp(sh.taken + (i & 1), ((i >> 1) & 1) ^ 1, &sh.abort);
      ct_fence();
      tc_fence_after();
      ct_products<CT_SV>(tmem + (uint32_t)((i & 1) * 4 * CT_SV), smem_u32(keys + place * CT_S_KEYS), CT_TERM,
                         CT_TILE, smem_u32(vals + (i & 1) * CT_S_VALS));
      umma_commit(sh.free + place);
      umma_commit(sh.done + (i & 1));
    }
  } else if (warp >= 8) {                                // ---- the values, weighted: lane = value size
    // (this warp's tokens of a chunk: two runs of eight, w and w + 4)
    const int w = warp - 8;
    uint8_t* mine = raw + w * (CT_S_RAW / 4);
    float2* mine_w = raw_w + w * 16;
    auto token = [&](int r) { return 8 * w + (r & 7) + (r >> 3) * 32; };
    auto fetch = [&](int i) {
      if (i < chunks) {
        uint8_t* to = mine + (i & 3) * CT_S_RAW;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int r = (lane >> 3) + 4 * x, t = i * CT_C + token(r);
          ds_cp16(reinterpret_cast<float*>(to + r * 128 + (lane & 7) * 16),
                  t < c.n ? vp + (size_t)t * p.v_stride + (lane & 7) * 4 : vsrc, t < c.n);
        }
        if (lane < 16) {
          const int t = i * CT_C + token(lane);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                           smem_u32(mine_w + (i & 3) * CT_C + lane)),
                       "l"(t < c.n ? wl + t : wl), "r"(t < c.n ? 8 : 0));
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = 0; i < 3; ++i) fetch(i);
    for (int i = 0; i < chunks; ++i) {
      __syncwarp();                                      // (all have read the place of chunk i - 1)
      fetch(i + 3);
      asm volatile("cp.async.wait_group 3;" ::: "memory");
      __syncwarp();
      if (i >= 2) ct_wait(sh.done + (i & 1), ((i >> 1) & 1) ^ 1, &sh.abort);
      const float* from = reinterpret_cast<const float*>(mine + (i & 3) * CT_S_RAW);
      const float2* from_w = mine_w + (i & 3) * CT_C;
      uint8_t* tile = vals + (i & 1) * CT_S_VALS;
      auto eight = [&](int x) {
        MtEight e;
#pragma unroll
        for (int j = 0; j < 8; ++j) e.v[j] = cs_times(from[(8 * x + j) * CT_SV + lane], from_w[8 * x + j]);
        return e;
      };
      float2 left = make_float2(0.f, 0.f);
#pragma unroll
      for (int x = 0; x < 2; ++x) mt_put(tile + mt_spot(lane, w + 4 * x), CT_SV * 128, eight(x), left);
      if (mt_bad(left)) {
#pragma unroll 1
        for (int x = 0; x < 2; ++x) {
          MtEight e = eight(x);
          if (mt_clean(e, MT_NO_TERMS_UP)) odd_v[i & 3][lane] = i + 1;
          mt_put(tile + mt_spot(lane, w + 4 * x), CT_SV * 128, e, left);
        }
      }
      ct_arrive(sh.put + (i & 1));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {                                               // ---- the state: key size k0 + own, 16 value sizes
    const int own = tid & 127, half = tid >> 7;
    const double* g = G + (size_t)h * p.T + c.t0;
    float* st = state + (size_t)slot * slot_stride + (size_t)h * p.dv * p.dk +
                (size_t)(v0 + 16 * half) * p.dk + k0 + own;
    const unsigned long long* odd_k = odd_rows + ((size_t)c.first * p.QH + hq) * 2 + 1;
    float* to = U + (((size_t)c.first * p.H + h) * p.dv + v0) * p.dk + (size_t)k0 * CT_SV;
    const size_t step = (size_t)p.H * p.dv * p.dk;
    const uint32_t from = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(16 * half);
    unsigned long long S[CT_SV / 4];
#pragma unroll
    for (int j = 0; j < CT_SV / 4; ++j) S[j] = cs_pair(st[(size_t)(2 * j) * p.dk], st[(size_t)(2 * j + 1) * p.dk]);
    float2 dec = make_float2(0.f, 0.f);                  // (lane l: over chunk l of the current 32)
    unsigned long long bad_k = odd_k[0];
    for (int i = 0; i < chunks; ++i) {
      if ((i & 31) == 0) {
        const int x = min(i + lane, chunks - 1);
        dec = cs_exp(g[min(c.n, (x + 1) * CT_C) - 1] - (x ? g[x * CT_C - 1] : 0.0));
      }
      const float dx = __shfl_sync(0xffffffffu, dec.x, i & 31), dy = __shfl_sync(0xffffffffu, dec.y, i & 31);
      // the state before the chunk leaves
      if (tid == 0) bf_bulk_wait_read<0>();
      asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
#pragma unroll
      for (int q = 0; q < CT_SV / 8; ++q) {
        float4 x;
        cs_unpair(S[2 * q], x.x, x.y);
        cs_unpair(S[2 * q + 1], x.z, x.w);
        *reinterpret_cast<float4*>(kept + own * CT_SV + (((q + 4 * half) ^ (own & 7)) << 2)) = x;
      }
      asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
      if (tid == 0) {
        ct_fence();
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(to + i * step),
                     "r"(smem_u32(kept)), "r"(128 * CT_SV * 4)
                     : "memory");
        bf_bulk_commit();
      }
      const unsigned long long bad_now = bad_k;
      if (i + 1 < chunks) bad_k = odd_k[(size_t)(i + 1) * p.QH * 2];
      ct_wait(sh.done + (i & 1), (i >> 1) & 1, &sh.abort);
      __syncwarp();
      tc_fence_after();
      // S <- last + (decay S + rest): where decays are fast the last tokens make up the state, rounded once
      unsigned long long was[CT_SV / 4], zero = 0ull;    // zero: NaN where some sum is not finite
      const bool second = c.n - i * CT_C > 32;
      const unsigned long long dx2 = cs_pair(dx, dx), dy2 = cs_pair(dy, dy), down = cs_pair(CT_DOWN, CT_DOWN);
#pragma unroll
      for (int j0 = 0; j0 < CT_SV / 4; j0 += 4) {
        unsigned long long last[4], rest[4];
        ct_take<CT_SV>(from + (uint32_t)((i & 1) * 4 * CT_SV + 2 * j0), second, last, rest);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          zero = cs_fma2(cs_add2(last[j], rest[j]), 0ull, zero);
          const unsigned long long before = S[j0 + j];
          was[j0 + j] = before;
          S[j0 + j] = cs_fma2(last[j], down, cs_fma2(dx2, before, cs_fma2(dy2, before, ct_mul2(rest[j], down))));
        }
      }
      // (ahead of the arrival: behind it the products of chunk i + 2 may be done and chunk i + 4's flag be put here)
      const bool odd = *(volatile int*)&odd_v[i & 3][lane] == i + 1;
      tc_fence_before();
      ct_arrive(sh.taken + (i & 1));
      float z0, z1;
      cs_unpair(zero, z0, z1);
      const bool lost = z0 + z1 != 0.f;
      const unsigned odd_cols = __ballot_sync(0xffffffffu, odd) >> (16 * half) & 0xffffu;
      if (odd_cols || bad_now || lost) {
        float again[CT_SV / 2];
        ct_state_again(qk + (size_t)(c.t0 + i * CT_C) * p.qk_stride + p.k_off + (size_t)hq * p.dk + k0 + own,
                       p.qk_stride, vp + (size_t)i * CT_C * p.v_stride + 16 * half, p.v_stride, wl + i * CT_C,
                       min(CT_C, c.n - i * CT_C), again);
#pragma unroll
        for (int j = 0; j < CT_SV / 4; ++j) {
          float x[2], b[2];
          cs_unpair(S[j], x[0], x[1]);
          cs_unpair(was[j], b[0], b[1]);
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (bad_now || (odd_cols >> (2 * j + e) & 1) || !(fabsf(x[e]) < INFINITY))
              x[e] = fmaf(dx, b[e], fmaf(dy, b[e], again[2 * j + e]));
          S[j] = cs_pair(x[0], x[1]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < CT_SV / 4; ++j) {
      float a, e;
      cs_unpair(S[j], a, e);
      st[(size_t)(2 * j) * p.dk] = a;
      st[(size_t)(2 * j + 1) * p.dk] = e;
    }
    if (tid == 0) bf_bulk_wait_read<0>();
  }
  ct_end<CT_S_COLS>(sh, tmem, warp, 13, err);
}

// ---------------------------------------------------------------------------------- ct_out
// Tiles of (chunk, 128 of the heads' value sizes side by side), dealt out to a CTA an SM.  The products' rows
// are value sizes, their columns the chunk's tokens: first the state times q over dk, a step of 64 at a time,
// times the token's weight, then the values times the weighted q . k; two heads of 64 have a step each there,
// whose sums only the lanes of that head add.
#define CT_O_A (3 * 2 * CT_TERM)                         // 64 terms x 128 value sizes in three terms
#define CT_O_SMEM (1024 + 2 * CT_O_A + 2 * CT_TILE + 2 * CT_TILE)
#define CT_O_COLS 512                                    // two places of 4 x 64 columns
// eight warps that add (a quarter of the lanes, half of the tokens each), eight that convert the states and values,
// four the weighted q . k, two that issue products and one that copies: 80 registers a thread at the start, 96, 80,
// 80 and 48 from then on.
// What every role does for a step is written once, rare paths are functions of their own: five roles' code,
// unrolled, was 158 KB, and warps waited for instructions most of their time (125 us).
#define CT_O_THREADS 768
#define CT_O_LIST 64                                     // most tiles of a CTA
template <int REGS>
__device__ __forceinline__ void ct_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS)); }
template <int REGS>
__device__ __forceinline__ void ct_fewer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS)); }

struct CtUnit {
  int col0, chunk, t0, n;                                // n: its tokens, 0: no such tile
  int h, hq;                                             // the (first) head, its q
};
// The results of the tokens in `again` (bits, from t_first on) for one value size by multiply-adds, in cs_out's
// order: runs of sixteen, the weight on q; four tokens at a time.  at: the tokens' weights, what is left of them
// CT_C floats behind.
__device__ __noinline__ void ct_out_again(const float* __restrict__ q, long long q_stride,
                                          const float* __restrict__ v, long long v_stride,
                                          const float* __restrict__ Pm, const float* __restrict__ S, int piece,
                                          int dk, const double* __restrict__ g, const double* __restrict__ hs,
                                          const float* at, int t_first, int n, unsigned again, float* dst,
                                          size_t row) {
#pragma unroll 1
  for (int t = 0; t < 32; t += 4) {
    if (!(again >> t & 15u)) continue;
    float o[4] = {0.f, 0.f, 0.f, 0.f};
    float2 w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = make_float2(at[t + j], at[CT_C + t + j]);
    const int last = min(t_first + t + 3, n - 1);
#pragma unroll 1
    for (int k0 = 0; k0 < dk; k0 += 16) {
      float run[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int k = k0; k < k0 + 16; ++k) {
        const float sv = S[(size_t)k * 32 + ((piece ^ (k & 7)) << 2)];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          run[j] = fmaf(cs_times(t_first + t + j < n ? q[(size_t)(t + j) * q_stride + k] : 0.f, w[j]), sv, run[j]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] += run[j];
    }
#pragma unroll 1
    for (int y0 = 0; y0 <= last; y0 += 16) {
      float run[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int y = y0; y <= min(last, y0 + 15); ++y) {
        const float vv = v[(size_t)y * v_stride];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (y <= t_first + t + j && t_first + t + j < n)
            run[j] = fmaf(cs_times(Pm[(t + j) * CT_C + y], cs_exp(g[t_first + t + j] - hs[y])), vv, run[j]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] += run[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (again >> (t + j) & 1u) dst[(size_t)(t + j) * row] = o[j];
  }
}
// A thread's four pieces of a step once more, with zeros where a number has no terms; which value sizes those are
// goes to `reach` (eight of them).
__device__ __noinline__ void ct_convert_again(const float* base, int stride, int o0, int o1, int rows,
                                              int row0, bool values, uint8_t* dst, int* reach, int tile) {
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    MtEight e = {};
    if (16 * i + row0 < rows) {
      const float4 a = *reinterpret_cast<const float4*>(base + i * stride + o0);
      const float4 b = *reinterpret_cast<const float4*>(base + i * stride + o1);
      e = {{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
    }
    const int bad = mt_clean(e, MT_NO_TERMS_UP);
    for (int j = 0; j < 8; ++j)
      if (bad >> j & 1) atomicMax(reach + j, tile * 64 + 63 - (values ? 16 * i + row0 : 0));
    float2 left = make_float2(0.f, 0.f);
    mt_put(dst + i * 16 * 128, 2 * CT_TERM, e, left);
  }
}

__global__ void __launch_bounds__(CT_O_THREADS, 1) ct_out_kernel(
    const float* __restrict__ qk, const float* __restrict__ vsrc, CsIn p, int n_chunks,
    const int* __restrict__ q_start, const int* __restrict__ state_slots, int n_slots,
    const double* __restrict__ G, const double* __restrict__ Hs, const CtHead* __restrict__ W,
    const float* __restrict__ qkm, const uint8_t* __restrict__ Xq,
    const unsigned long long* __restrict__ odd_rows, const float* __restrict__ U, float* __restrict__ o_raw,
    int* __restrict__ err) {
  extern __shared__ __align__(16) uint8_t ct_raw[];
  __shared__ CtShared sh;
  __shared__ CtUnit list[CT_O_LIST];                     // the CTA's tiles, in order
  // [tile % 4][head] the tokens' weights of the state before, and what is left of them
  __shared__ __align__(16) float at_s[4][2][2][CT_C];
  // (of tile % 4; tile counted from 1) tile * 64 + 63 - the first token that a value size without terms reaches;
  // tile: the token's weighted q . k has no terms
  __shared__ int odd_m[4][128], odd_t[4][2][CT_C];
  uint8_t* a_ring = ct_raw + ((1024u - (smem_u32(ct_raw) & 1023u)) & 1023u);
  uint8_t* q_ring = a_ring + 2 * CT_O_A;
  uint8_t* w_ring = q_ring + 2 * CT_TILE;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int vtiles = p.H * p.dv / 128, steps = p.dk / 64, heads = p.dv < 128 ? 2 : 1, group = p.H / p.QH;
  const int units = n_chunks * vtiles;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(sh.full + i, 1);
      mbar_init(sh.free + i, 1);
      mbar_init(sh.put + i, 8);
      mbar_init(sh.a_free + i, heads);
      mbar_init(sh.w_put + i, 4);
      mbar_init(sh.w_free + i, 1);
      mbar_init(sh.done + i, 1);
      mbar_init(sh.taken + i, 8);
    }
    mbar_init(&sh.drain, 2);
    sh.abort = 0;
  }
  for (int i = tid; i < 4 * 128; i += CT_O_THREADS) {
    odd_m[i / 128][i % 128] = 0;
    odd_t[i / 128][i / 64 % 2][i % 64] = 0;
  }
  for (int i = tid; i < 2 * CT_TILE / 16; i += CT_O_THREADS)       // (q . k above the diagonal stays zero)
    reinterpret_cast<uint4*>(w_ring)[i] = make_uint4(0, 0, 0, 0);
  // tiles of a chunk one after the other, so that the CTAs which share it run together; at most CT_O_LIST of them
  const int own_units = (units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  for (int i = warp; i < own_units; i += CT_O_THREADS / 32) {
    const int u = blockIdx.x + i * gridDim.x;
    CtUnit x;
    x.col0 = u % vtiles * 128;
    x.chunk = u / vtiles;
    const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, x.chunk, -1);
    const int slot = c.b < 0 ? -1 : state_slots[c.b];
    x.t0 = c.t0 + c.index * CT_C;
    x.n = slot < 0 || slot >= n_slots ? 0 : min(CT_C, c.n - c.index * CT_C);
    x.h = x.col0 / p.dv;
    x.hq = x.h / group;
    if (lane == 0) list[i] = x;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  const uint32_t tmem = ct_begin<CT_O_COLS>(sh, warp, 20);

  if (warp >= 20) {
    ct_fewer<48>();
    if (warp == 22) {                                    // ---- q's tiles
      if (lane == 0) {
        int place = 0, i = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int k = 0; k < own_units && ok; ++k) {
          if (list[k].n == 0) continue;
          const uint8_t* X = Xq + ((size_t)list[k].chunk * p.QH + list[k].hq) * steps * CT_TILE;
          for (int s = 0; s < steps; ++s, ++i) {
            ok = i < 2 || ct_wait(sh.free + place, phase ^ 1u, &sh.abort);
            if (!ok) break;
            mbar_expect_tx(sh.full + place, CT_TILE);
            bf_bulk_load(q_ring + place * CT_TILE, X + (size_t)s * CT_TILE, CT_TILE, sh.full + place);
            if (++place == 2) place = 0, phase ^= 1u;
          }
        }
        if (*(volatile int*)&sh.abort) mbar_drain(sh.full, 2, place, phase);
      }
      __syncwarp();
    } else if (warp < 22) {                              // ---- products: steps in turn
      int iq = 0, ia = 0, iw = 0, is = 0;                // tiles of q, rows, weighted q . k, sums
      for (int k = 0; k < own_units; ++k) {
        if (list[k].n == 0) continue;
#pragma unroll 1
        for (int s = 0; s < steps + heads; ++s, ++is) {
          const bool of_q = s < steps, next_a = of_q || s + 1 == steps + heads;
          const int ib = of_q ? iq++ : iw++;
          if ((is & 1) == warp - 20) {
            ct_wait_warp((of_q ? sh.full : sh.w_put) + (ib & 1), (ib >> 1) & 1, &sh.abort);
            ct_wait_warp(sh.put + (ia & 1), (ia >> 1) & 1, &sh.abort);
            if (is >= 2) ct_wait_warp(sh.taken + (is & 1), ((is >> 1) & 1) ^ 1, &sh.abort);
            ct_fence();
            tc_fence_after();
            ct_products<CT_C>(tmem + (uint32_t)((is & 1) * 4 * CT_C), smem_u32(a_ring + (ia & 1) * CT_O_A),
                              2 * CT_TERM, CT_TERM, smem_u32((of_q ? q_ring : w_ring) + (ib & 1) * CT_TILE));
            umma_commit((of_q ? sh.free : sh.w_free) + (ib & 1));
            umma_commit(sh.a_free + (ia & 1));           // (the values' place is free behind both heads' steps)
            if (of_q && heads == 2) umma_commit(sh.a_free + (ia & 1));
            umma_commit(sh.done + (is & 1));
          }
          if (next_a) ++ia;
        }
      }
    }
  } else if (warp >= 16) {                               // ---- the weighted q . k's terms
    // ten pieces of 16 rows x 16 columns (row block, column block), two or three of them a warp's: a thread has
    // row lane / 2 and eight columns
    const int w = warp - 16, ops = w < 2 ? 3 : 2;
    auto rows_of = [&](int j) { return w == 0 ? 3 : w == 1 ? 2 : w == 2 ? (j ? 0 : 3) : 1; };
    auto cols_of = [&](int j) { return w == 2 ? (j ? 0 : 3) : j; };
    int k = 0, head = 0, tile = 1;
    while (k < own_units && list[k].n == 0) ++k;
    float4 P[3][2];
    float at = 0.f;
    const CtHead* from = W;
    auto source = [&]() { from = W + (size_t)list[k].chunk * p.H + list[k].h + head; };
    auto fetch = [&](int j) {
      if (k >= own_units || j >= ops) return;
      const float4* s =
          reinterpret_cast<const float4*>(&from->P[16 * rows_of(j) + (lane >> 1)][16 * cols_of(j) + 8 * (lane & 1)]);
      P[j][0] = s[0];
      P[j][1] = s[1];
    };
    if (k < own_units) {
      source();
      at = from->at[w >> 1][(w & 1) * 32 + lane];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) fetch(j);
#pragma unroll 1
    for (int iw = 0; k < own_units; ++iw) {
      const int place = iw & 1, tag = tile, at_head = head;
      if (++head == heads) {
        head = 0;
        ++tile;
        do ++k;
        while (k < own_units && list[k].n == 0);
      }
      if (iw >= 2) ct_wait(sh.w_free + place, ((iw >> 1) & 1) ^ 1, &sh.abort);
      __syncwarp();
      at_s[tag & 3][at_head][w >> 1][(w & 1) * 32 + lane] = at;
      if (k < own_units) {
        source();
        at = from->at[w >> 1][(w & 1) * 32 + lane];
      }
      uint8_t* tw = w_ring + place * CT_TILE;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        if (j >= ops) continue;
        const MtEight e = {{P[j][0].x, P[j][0].y, P[j][0].z, P[j][0].w, P[j][1].x, P[j][1].y, P[j][1].z, P[j][1].w}};
        fetch(j);
        const int t = 16 * rows_of(j) + (lane >> 1);
        float2 left = make_float2(0.f, 0.f);
        uint8_t* dst = tw + mt_spot(t, 2 * cols_of(j) + (lane & 1));
        mt_put(dst, CT_TERM, e, left);
        if (mt_bad(left)) {                              // (the row is computed by multiply-adds)
          odd_t[tag & 3][at_head][t] = tag;
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(dst + i * CT_TERM) = make_uint4(0, 0, 0, 0);
        }
      }
      ct_arrive(sh.w_put + place);
    }
  } else if (warp >= 8) {                                // ---- the state's and the values' terms
    // a piece of eight value sizes: block of 32 (cw % 4), octet lane % 4; rows 16 i + 8 (cw / 4) + r
    const int cw = warp - 8, vb = cw & 3, q4 = lane & 3, r = ((lane >> 2) & 1) * 4 + (lane >> 3);
    const int row0 = (cw >> 2) * 8 + r;
    uint8_t* spot = a_ring + (vb >> 1) * CT_TERM + mt_spot(row0, (vb & 1) * 4 + q4);
    // a step's source: from row to row 16 further, the two halves of a piece, how many rows there are
    const float* base = nullptr;
    int stride = 0;
    int o[2] = {0, 0}, rows = 0;
    int k = 0, s = 0;                                    // (of the step whose numbers are asked for)
    while (k < own_units && list[k].n == 0) ++k;
    auto source = [&]() {
      if (s == 0) {
        base = U + ((size_t)list[k].chunk * p.H * p.dv + list[k].col0 + vb * 32) * p.dk + row0 * 32;
        stride = 16 * 32;
        o[0] = ((2 * q4) ^ r) << 2;
        o[1] = ((2 * q4 + 1) ^ r) << 2;
        rows = 64;
      } else if (s < steps) {
        base += 64 * 32;
      } else {
        base = vsrc + (size_t)(list[k].t0 + row0) * p.v_stride + p.v_off + list[k].col0 + vb * 32 + q4 * 8;
        stride = 16 * (int)p.v_stride;
        o[0] = 0;
        o[1] = 4;
        rows = list[k].n;
      }
    };
    float4 f[4][2];
    auto fetch = [&](int i) {
      if (16 * i + row0 < rows) {
        f[i][0] = *reinterpret_cast<const float4*>(base + (i * stride + o[0]));
        f[i][1] = *reinterpret_cast<const float4*>(base + (i * stride + o[1]));
      } else {
        f[i][0] = f[i][1] = cs_zero();
      }
    };
    if (k < own_units) {
      source();
#pragma unroll
      for (int i = 0; i < 4; ++i) fetch(i);
    }
    int tile = 1;
#pragma unroll 1
    for (int ia = 0; k < own_units; ++ia) {
      const float* was = base;
      const int was_stride = stride, was0 = o[0], was1 = o[1], was_rows = rows, was_tile = tile;
      const bool values = s == steps;
      if (++s > steps) {
        s = 0;
        ++tile;
        do ++k;
        while (k < own_units && list[k].n == 0);
      }
      if (k < own_units) source();
      else rows = 0;
      if (ia >= 2) ct_wait(sh.a_free + (ia & 1), ((ia >> 1) & 1) ^ 1, &sh.abort);
      __syncwarp();
      uint8_t* dst = spot + (ia & 1) * CT_O_A;
      float2 left = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const MtEight e = {{f[i][0].x, f[i][0].y, f[i][0].z, f[i][0].w, f[i][1].x, f[i][1].y, f[i][1].z, f[i][1].w}};
        fetch(i);
        mt_put(dst + i * 16 * 128, 2 * CT_TERM, e, left);
      }
      if (mt_bad(left))
        ct_convert_again(was, was_stride, was0, was1, was_rows, row0, values, dst,
                         &odd_m[was_tile & 3][vb * 32 + q4 * 8], was_tile);
      ct_arrive(sh.put + (ia & 1));
    }
  } else {                                               // ---- sums: value size m, tokens t_first ..
    ct_more<96>();
    const int quarter = warp & 3, t_first = (warp >> 2) * 32, m = quarter * 32 + lane;
    const int own = heads == 2 ? quarter >> 1 : 0;       // which of the tile's heads
    const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)t_first;
    const size_t row = (size_t)p.H * p.dv;
    int is = 0, tile = 1;
#pragma unroll 1
    for (int k = 0; k < own_units; ++k) {
      const CtUnit x = list[k];
      if (x.n == 0) continue;
      unsigned long long sum[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) sum[j] = 0ull;
      const float* at = at_s[tile & 3][own][0] + t_first;
      float* dst = o_raw + (size_t)x.t0 * row + (size_t)t_first * row + x.col0 + m;
      const int n = x.n - t_first;
#pragma unroll 1
      for (int s = 0; s < steps + heads; ++s, ++is) {
        ct_wait(sh.done + (is & 1), (is >> 1) & 1, &sh.abort);
        __syncwarp();
        tc_fence_after();
        if (s < steps) {
#pragma unroll
          for (int j0 = 0; j0 < 16; j0 += 4) {
            unsigned long long last[4], rest[4];
            ct_take<CT_C>(from + (uint32_t)((is & 1) * 4 * CT_C + 2 * j0), t_first > 0, last, rest);
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[j0 + j] = cs_add2(sum[j0 + j], cs_add2(last[j], rest[j]));
          }
        } else if (s - steps == own) {                   // (the weights were there before that step's q . k)
#pragma unroll
          for (int j0 = 0; j0 < 16; j0 += 4) {
            unsigned long long last[4], rest[4];
            ct_take<CT_C>(from + (uint32_t)((is & 1) * 4 * CT_C + 2 * j0), t_first > 0, last, rest);
#pragma unroll
            for (int j = j0; j < j0 + 4; ++j) {
              const unsigned long long w = *reinterpret_cast<const unsigned long long*>(at + 2 * j);
              const unsigned long long wl = *reinterpret_cast<const unsigned long long*>(at + CT_C + 2 * j);
              sum[j] = cs_add2(cs_add2(cs_fma2(sum[j], w, ct_mul2(sum[j], wl)), rest[j - j0]), last[j - j0]);
              float a, b;
              cs_unpair(ct_mul2(sum[j], CT_DOWN), a, b);
              if (2 * j < n) dst[(size_t)(2 * j) * row] = a;
              if (2 * j + 1 < n) dst[(size_t)(2 * j + 1) * row] = b;
            }
          }
        }
        tc_fence_before();
        ct_arrive(sh.taken + (is & 1));
      }
      unsigned long long zero = 0ull;                    // (NaN where some sum is not finite)
#pragma unroll
      for (int j = 0; j < 16; ++j) zero = cs_fma2(sum[j], 0ull, zero);
      float z0, z1;
      cs_unpair(zero, z0, z1);
      unsigned again = 0u;                               // tokens whose sum is not finite, or not of terms
      if (z0 + z1 != 0.f) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float a, b;
          cs_unpair(sum[j], a, b);
          again |= (fabsf(a) < INFINITY ? 0u : 1u << (2 * j)) | (fabsf(b) < INFINITY ? 0u : 2u << (2 * j));
        }
      }
      const int h = x.h + own, hq = x.hq;
      again |= (unsigned)(odd_rows[((size_t)x.chunk * p.QH + hq) * 2] >> t_first);
      const int reach = *(volatile int*)&odd_m[tile & 3][m];
      if (reach >> 6 == tile) {                          // from its first token on
        const int first = 63 - (reach & 63) - t_first;
        again |= first <= 0 ? 0xffffffffu : first < 32 ? 0xffffffffu << first : 0u;
      }
      again |= __ballot_sync(0xffffffffu, *(volatile int*)&odd_t[tile & 3][own][t_first + lane] == tile);
      if (n < 32) again &= n > 0 ? (1u << n) - 1u : 0u;
      if (again)
        ct_out_again(qk + (size_t)(x.t0 + t_first) * p.qk_stride + p.q_off + (size_t)hq * p.dk, p.qk_stride,
                     vsrc + (size_t)x.t0 * p.v_stride + p.v_off + x.col0 + m, p.v_stride,
                     qkm + (((size_t)x.chunk * p.QH + hq) * CT_C + t_first) * CT_C,
                     U + ((size_t)x.chunk * p.H * p.dv + x.col0 + (m & ~31)) * p.dk + (m & 3), (m & 31) >> 2, p.dk,
                     G + (size_t)h * p.T + x.t0, Hs + (size_t)h * p.T + x.t0, at, t_first, x.n, again, dst, row);
      __syncwarp();
      ++tile;
    }
  }
  ct_end<CT_O_COLS>(sh, tmem, warp, 20, err);
}

// -------------------------------------------------------------------------------- dt_walk
// The delta rule's chain from chunk to chunk (ds_walk) with keys of 128: U = Y - W S, S <- exp(F_C) S + K^T
// (exp(F_C - F) U).  grid (32 value sizes, H, B).  Eight warps keep 128 x 32 of the state, half a row a thread, and
// take each product's operand apart as the other's sums come; one warp issues products, one asks for W's and K's
// tiles (X: W in terms, chunk and head by chunk and head).  The state before a chunk leaves as ct_state's does.
//
// W S: 64 tokens x 32 columns over 128 terms, leading terms' products summed 32 at a time (four places), the
// others' in two; a warp reads its 16 rows in the shape of a fragment, rows lane / 4 and eight further, so that
// neighbouring tokens, which lie side by side in the next operand, are one exchange away.
#define DT_TERM (CT_SV * 128)                            // 32 columns x 64 terms
#define DT_SMEM (1024 + 2 * CT_S_KEYS + 9 * DT_TERM + 128 * CT_SV * 4 + CT_C * CT_SV * 4)
#define DT_THREADS 320
#define DT_SUMS 192                                      // columns of W S's places; K^T U's four of 32 behind them

// rows' terms K-major (two tiles of 64 sizes) times columns' (two tiles of 32 x 64)
__device__ __forceinline__ void dt_products(uint32_t d, uint32_t a, uint32_t b) {
  constexpr uint32_t base = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(64 >> 4) << 24);
  constexpr uint32_t one = base | ((uint32_t)(32 >> 3) << 17), two = base | ((uint32_t)(64 >> 3) << 17),
                     three = base | ((uint32_t)(96 >> 3) << 17);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t ak = a + (k >> 2) * CT_TILE + (k & 3) * 32, bk = b + (k >> 2) * 3 * DT_TERM + (k & 3) * 32;
    const uint64_t hi = umma_desc_k_sw128(ak), mid = umma_desc_k_sw128(ak + CT_TERM),
                   lo = umma_desc_k_sw128(ak + 2 * CT_TERM), bh = umma_desc_k_sw128(bk),
                   bm = umma_desc_k_sw128(bk + DT_TERM);
    if (k < 2) {
      umma_bf16(d, hi, bh, three, k > 0);
    } else {
      umma_bf16(d + 64 + (k >> 1) * 32, hi, bh, one, k & 1);
      umma_bf16(d + 32, hi, bm, two, 1);
    }
    umma_bf16(d + 32, mid, bh, two, 1);
    umma_bf16(d + 64, lo, bh, one, 1);
  }
}
__device__ __forceinline__ void dt_load(uint32_t at, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(at));
}
// Two neighbouring numbers of a row of terms, times SPLIT_UP, to `at` (a term's tile DT_TERM behind the one
// before); numbers without terms as zeros, and true
__device__ __forceinline__ bool dt_put(uint8_t* at, float a, float b) {
  const bool bad_a = (__float_as_uint(a) & 0x7fffffffu) >= CS_NO_TERMS_UP,
             bad_b = (__float_as_uint(b) & 0x7fffffffu) >= CS_NO_TERMS_UP;
  if (bad_a) a = 0.f;
  if (bad_b) b = 0.f;
  uint32_t hi, mid, lo;
  split_up(a, b);
  split3(a, b, hi, mid, lo);
  *reinterpret_cast<uint32_t*>(at) = hi;
  *reinterpret_cast<uint32_t*>(at + DT_TERM) = mid;
  *reinterpret_cast<uint32_t*>(at + 2 * DT_TERM) = lo;
  return bad_a || bad_b;
}
// W S of two rows and their four columns (8 c + col, + 1) by multiply-adds, in ds_walk's order
__device__ __noinline__ void dt_again_ws(const float* w0, const float* w1, const float* kept, int col, float* out) {
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int k0 = 0; k0 < 128; k0 += 16) {
      float run[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int k = k0; k < k0 + 16; ++k) {
        const int v = 8 * c + col;
        const float2 x = *reinterpret_cast<const float2*>(kept + k * CT_SV + (((v >> 2) ^ (k & 7)) << 2) + (v & 3));
        run[0] = fmaf(w0[k], x.x, run[0]);
        run[1] = fmaf(w0[k], x.y, run[1]);
        run[2] = fmaf(w1[k], x.x, run[2]);
        run[3] = fmaf(w1[k], x.y, run[3]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] += run[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) out[4 * c + j] = o[j];
  }
}
// half a row of the state behind the chunk by multiply-adds, one chain a number
__device__ __noinline__ void dt_again_state(const float* k, long long k_stride, const float* us, int n, float2 g,
                                            const float* was, float* out) {
#pragma unroll 1
  for (int j = 0; j < CT_SV / 2; ++j) {
    float x = cs_times(was[j], g);
#pragma unroll 4
    for (int s = 0; s < n; ++s) x = fmaf(k[(size_t)s * k_stride], us[s * CT_SV + j], x);
    out[j] = x;
  }
}

__global__ void __launch_bounds__(DT_THREADS, 1) dt_walk_kernel(
    DsIn p, const int* __restrict__ q_start, const int* __restrict__ state_slots, int n_slots,
    float* __restrict__ state, long long slot_stride, const double* __restrict__ F,
    const float2* __restrict__ Wl, const float* __restrict__ W, const float* __restrict__ Y,
    const uint8_t* __restrict__ Xw, const unsigned long long* __restrict__ odd_w, const uint8_t* __restrict__ Xk,
    const unsigned long long* __restrict__ odd_rows, float* __restrict__ u, float* __restrict__ Sc,
    int* __restrict__ err) {
  extern __shared__ __align__(16) uint8_t ct_raw[];
  __shared__ CtShared sh;                                // full, free: W's and K's tiles; put, done: S's, U's
  __shared__ int odd_s[2];                               // of S and of U: chunk + 1 where a number has no terms
  uint8_t* w_tile = ct_raw + ((1024u - (smem_u32(ct_raw) & 1023u)) & 1023u);
  uint8_t* k_tile = w_tile + CT_S_KEYS;
  uint8_t* s_op = k_tile + CT_S_KEYS;                    // two tiles of three terms
  uint8_t* u_op = s_op + 6 * DT_TERM;
  float* kept = reinterpret_cast<float*>(u_op + 3 * DT_TERM);            // [128][32]
  float* us = kept + 128 * CT_SV;                        // [64][32]
  const int h = blockIdx.y, b = blockIdx.z, col0 = blockIdx.x * CT_SV;
  const CsChunk c = cs_find(q_start, p.B, CT_C, p.n_min, 0, b);
  if (c.n <= p.n_min) return;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= n_slots) {
    if (threadIdx.x == 0) atomicOr(err, BF_ERR_SLOT);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hq = h / (p.H / p.G), chunks = (c.n + CT_C - 1) / CT_C;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(sh.full + i, 1);
      mbar_init(sh.free + i, 1);
      mbar_init(sh.put + i, 8);
      mbar_init(sh.done + i, 1);
      odd_s[i] = 0;
    }
    mbar_init(&sh.drain, 2);
    sh.abort = 0;
  }
  const uint32_t tmem = ct_begin<512>(sh, warp, 8);

  if (warp == 9) {                                       // ---- tiles; (also of the second warp that ct_end expects)
    if (lane == 0) {
      uint32_t phase = 0;
      bool ok = true;
      int asked = 0;                                     // fills of both places in turn
      for (int i = 0; i < chunks && ok; ++i, phase ^= 1u) {
        const size_t chunk = (size_t)(c.first + i);
        for (int x = 0; x < 2 && ok; ++x) {
          ok = i == 0 || ct_wait(sh.free + x, phase ^ 1u, &sh.abort);
          if (!ok) break;
          mbar_expect_tx(sh.full + x, CT_S_KEYS);
          bf_bulk_load(x ? k_tile : w_tile,
                       x ? Xk + (chunk * p.G + hq) * CT_S_KEYS : Xw + (chunk * p.H + h) * CT_S_KEYS, CT_S_KEYS,
                       sh.full + x);
          ++asked;
        }
      }
      if (*(volatile int*)&sh.abort) mbar_drain(sh.full, 2, asked & 1, (uint32_t)(asked >> 1) & 1u);
    }
    __syncwarp();
  } else if (warp == 8) {                                // ---- products
    for (int i = 0; i < chunks; ++i) {
      ct_wait_warp(sh.full, i & 1, &sh.abort);
      ct_wait_warp(sh.put, i & 1, &sh.abort);
      ct_fence();
      tc_fence_after();
      dt_products(tmem, smem_u32(w_tile), smem_u32(s_op));
      umma_commit(sh.done);
      umma_commit(sh.free);
      ct_wait_warp(sh.full + 1, i & 1, &sh.abort);
      ct_wait_warp(sh.put + 1, i & 1, &sh.abort);
      ct_fence();
      tc_fence_after();
      ct_products<CT_SV>(tmem + DT_SUMS, smem_u32(k_tile), CT_TERM, CT_TILE, smem_u32(u_op));
      umma_commit(sh.done + 1);
      umma_commit(sh.free + 1);
    }
  } else {
    const int own = tid & 127, half = tid >> 7, quarter = warp & 3;        // key size; columns 16 half ..
    float* st = state + (size_t)slot * slot_stride + ((size_t)h * p.dv + col0 + 16 * half) * 128 + own;
    const double* f = F + (size_t)h * p.T + c.t0;
    const float2* wl = Wl + (size_t)h * p.T + c.t0;
    const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(16 * half);
    // of W S: rows 16 quarter + r, + 8, columns q + 8 c, + 1
    const int r = lane >> 2, q = 16 * half + 2 * (lane & 3), t_own = 16 * quarter + r;
    float S[CT_SV / 2];
#pragma unroll
    for (int j = 0; j < CT_SV / 2; ++j) S[j] = st[(size_t)j * 128];
    double before = 0.0;
    for (int i = 0; i < chunks; ++i) {
      const int n = min(CT_C, c.n - i * CT_C);
      const size_t chunk = (size_t)(c.first + i) * p.H + h;
      const float* y_at = Y + (chunk * CT_C + t_own) * p.dv + col0 + q;
      float2 y[2][2], g_t[2];                            // (asked for ahead of the products that need them)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
#pragma unroll
        for (int j = 0; j < 2; ++j) y[x][j] = *reinterpret_cast<const float2*>(y_at + (size_t)(8 * x) * p.dv + 8 * j);
        const int t = t_own + 8 * x;
        g_t[x] = t < n ? wl[i * CT_C + t] : make_float2(0.f, 0.f);
      }
      const unsigned long long bad_w = odd_w[chunk], bad_k = odd_rows[((size_t)(c.first + i) * p.G + hq) * 2 + 1];
      const double last = f[i * CT_C + n - 1];
      // ---- the state: as it is, and in terms
      if (tid == 0) bf_bulk_wait_read<0>();
      asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
#pragma unroll
      for (int x = 0; x < CT_SV / 8; ++x)
        *reinterpret_cast<float4*>(kept + own * CT_SV + (((x + 4 * half) ^ (own & 7)) << 2)) =
            make_float4(S[4 * x], S[4 * x + 1], S[4 * x + 2], S[4 * x + 3]);
      {
        // keys own and its neighbour: the even one takes the first eight columns of both
        const bool second = own & 1;
        uint8_t* to = s_op + (own >> 6) * 3 * DT_TERM + (own & 6) * 2 + 16 * half * 128;
        const int piece = (own & 63) >> 3;
        bool bad = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float keep = second ? S[j + 8] : S[j], give = second ? S[j] : S[j + 8];
          const float got = __shfl_xor_sync(0xffffffffu, give, 1);
          const int v = j + (second ? 8 : 0);
          bad |= dt_put(to + v * 128 + ((piece ^ (j & 7)) << 4), second ? got : keep, second ? keep : got);
        }
        if (bad) odd_s[0] = i + 1;
      }
      ct_arrive(sh.put);
      asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
      if (tid == 0) {
        ct_fence();
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                         Sc + (chunk * p.dv + col0) * 128),
                     "r"(smem_u32(kept)), "r"(128 * CT_SV * 4)
                     : "memory");
        bf_bulk_commit();
      }
      const float2 g = cs_exp(last - before);
      before = last;
      // ---- U
      ct_wait(sh.done, i & 1, &sh.abort);
      __syncwarp();
      tc_fence_after();
      float a[8];                                        // [column block][row, column]: rows t_own, + 8
      {
        uint32_t x0[8], x1[8], x2[8], x3[8], x4[8], x5[8];
        dt_load(from, x0);
        dt_load(from + 96, x1);
        dt_load(from + 128, x2);
        dt_load(from + 160, x3);
        dt_load(from + 32, x4);
        dt_load(from + 64, x5);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float lead = (__uint_as_float(x0[j]) + __uint_as_float(x1[j])) +
                             (__uint_as_float(x2[j]) + __uint_as_float(x3[j]));
          a[j] = (lead + (__uint_as_float(x4[j]) + __uint_as_float(x5[j]))) * CT_DOWN;
        }
      }
      float zero = 0.f;                                  // (NaN where some sum is not finite)
#pragma unroll
      for (int j = 0; j < 8; ++j) zero = fmaf(a[j], 0.f, zero);
      const bool odd = *(volatile int*)&odd_s[0] == i + 1;
      if (odd || (bad_w >> t_own & 0x101ull) || zero != 0.f) {
        float again[8];
        dt_again_ws(W + (chunk * CT_C + t_own) * 128, W + (chunk * CT_C + t_own + 8) * 128, kept, q, again);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (odd || (bad_w >> (t_own + (j & 2) * 4) & 1ull) || !(fabsf(a[j]) < INFINITY)) a[j] = again[j];
      }
      bool bad = false;
      {
        // tokens t_own and its neighbour (lane ^ 4): the even one takes the first column of both
        const bool second = r & 1;
        float* u_at = u + ((size_t)(c.t0 + i * CT_C + t_own) * p.H + h) * p.dv + col0 + q;
        uint8_t* to = u_op + (q + second) * 128 + (r & 6) * 2;
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float2 uv = make_float2(y[x][j].x - a[4 * j + 2 * x], y[x][j].y - a[4 * j + 2 * x + 1]);
            if (t_own + 8 * x < n)
              *reinterpret_cast<float2*>(u_at + (size_t)(8 * x) * p.H * p.dv + 8 * j) = uv;
            const float2 w = make_float2(cs_times(uv.x, g_t[x]), cs_times(uv.y, g_t[x]));
            *reinterpret_cast<float2*>(us + (t_own + 8 * x) * CT_SV + 8 * j + q) = w;
            const float keep = second ? w.y : w.x, got = __shfl_xor_sync(0xffffffffu, second ? w.x : w.y, 4);
            bad |= dt_put(to + 8 * j * 128 + (((2 * quarter + x) ^ ((q + second) & 7)) << 4), second ? got : keep,
                          second ? keep : got);
          }
        if (bad) odd_s[1] = i + 1;
      }
      tc_fence_before();
      ct_arrive(sh.put + 1);
      // ---- the state behind the chunk
      ct_wait(sh.done + 1, i & 1, &sh.abort);
      __syncwarp();
      tc_fence_after();
      float now[CT_SV / 2], z = 0.f;                         // z: NaN where some sum is not finite
#pragma unroll
      for (int j0 = 0; j0 < CT_SV / 4; j0 += 4) {
        unsigned long long x[4], y[4];
        ct_take<CT_SV>(from + DT_SUMS + (uint32_t)(2 * j0), n > 32, x, y);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float l[2], m[2];
          cs_unpair(x[j], l[0], l[1]);
          cs_unpair(ct_mul2(y[j], CT_DOWN), m[0], m[1]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {                  // (as in ct_state)
            const float was = S[2 * (j0 + j) + e];
            now[2 * (j0 + j) + e] = fmaf(l[e], CT_DOWN, fmaf(g.x, was, fmaf(g.y, was, m[e])));
            z = fmaf(l[e] + m[e], 0.f, z);
          }
        }
      }
      tc_fence_before();
      if (*(volatile int*)&odd_s[1] == i + 1 || bad_k || z != 0.f) {
        // (all rows of us are there: their products are)
        float was[CT_SV / 2], again[CT_SV / 2];
#pragma unroll
        for (int j = 0; j < CT_SV / 2; ++j) was[j] = S[j];
        dt_again_state(p.qkv + (size_t)(c.t0 + i * CT_C) * p.stride + (size_t)(p.G + hq) * 128 + own, p.stride,
                       us + 16 * half, n,
                       g, was, again);
#pragma unroll
        for (int j = 0; j < CT_SV / 2; ++j) now[j] = again[j];
      }
#pragma unroll
      for (int j = 0; j < CT_SV / 2; ++j) S[j] = now[j];
    }
#pragma unroll
    for (int j = 0; j < CT_SV / 2; ++j) st[(size_t)j * 128] = S[j];
    if (tid == 0) bf_bulk_wait_read<0>();
  }
  ct_end<512>(sh, tmem, warp, 8, err);
}

// Chunks of 64, keys in whole steps of 128, values of 64 or in whole tiles of 128 (two heads of 64 share a
// tile: an even number of them, reading the same q).
static bool ct_takes(int H, int QH, int dk, int dv, int C, int chunks) {
  return C == CT_C && dk % 128 == 0 && (dv % 128 == 0 || (dv == 64 && (H / QH) % 2 == 0)) &&
         (long long)chunks * H * dv < 0x7fffffff;
}
static size_t ct_terms_bytes(int chunks, int QH, int dk) {       // of q or k
  return (size_t)chunks * QH * (dk / 64) * CT_TILE;
}
static int ct_configure() {
  static bool configured_on[BF_MAX_DEVICES];
  bool& configured = configured_on[bf_current_device()];
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(ct_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         CT_S_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ct_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CT_O_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(dt_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return 0;
}
static void ct_out_launch(const float* qk, const float* v, const CsIn& p, int chunks, const int* q_start,
                          const int* state_slots, int n_slots, const double* G, const double* Hs,
                          const CtHead* W, const float* qkm, const uint8_t* Xq, const unsigned long long* odd,
                          const float* U, float* o_raw, int* err, cudaStream_t stream) {
  const long long units = (long long)chunks * (p.H * p.dv / 128);
  // (a CTA an SM; more of them where one's list would get too long)
  const long long most = (units + CT_O_LIST - 1) / CT_O_LIST;
  const unsigned grid = (unsigned)(most > 148 ? most : units < 148 ? units : 148);
  ct_out_kernel<<<grid, CT_O_THREADS, CT_O_SMEM, stream>>>(
      qk, v, p, chunks, q_start, state_slots, n_slots, G, Hs, W, qkm, Xq, odd, U, o_raw, err);
}
