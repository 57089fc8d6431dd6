// Causal grouped attention over the pages for the float32 engine, prompt portions and single tokens
// alike (heads of 64 or 128, no changes to the scores; attention_generic.cu takes the rest).
//
// A row is a (token, head of one kv head's group) pair, tokens in order.  A CTA takes BM rows of one
// (request, kv head) and walks the keys in tiles of 64 whose edges lie at multiples of 64 of the
// position; K and V tiles arrive by asynchronous copies a tile ahead.  Thread (tx, ty) of 16 x BM / TM
// has rows ty TM .. and keys tx + 16 j of the tile: q . k over pairs of sizes (even and odd terms in
// the two halves of packed multiply-adds, added at the end), the row's maximum and sum over the
// sixteen threads of a row by shuffles, then columns 4 tx + 64 j of O += P V.  FP32 multiply-adds
// throughout (fma.rn.f32x2).
//
// Every sum has an order that depends on the row's own position alone: a tile that a row does not see
// multiplies its sums by one and adds zeros.  So a row's result does not depend on how a prompt was
// cut, on BM, or on what else is in the batch.  A value that is not finite would make such a zero NaN:
// tiles of which a row sees a part only are looked through for one, and if there is, they are added
// key by key, each row its own.
//
// What bounds it: the FP32 pipes and, for them, shared-memory reads (one 16-byte read per eight
// multiply-adds).  The kernel for any size has one warp per (token, head), whose lanes share a key's
// sizes and meet in five shuffles per key: 333 tokens of 16 heads of 128 took 557 us there, 38 here (one
// token behind 499: 324 and 34).  With a page lookup for every 16-byte piece instead of every row these were
// 60 and 72.
#include <float.h>

#include "common.cuh"
#include "mma_utils.cuh"

#define AF_KEYS 64

__device__ __forceinline__ unsigned long long af_fma2(unsigned long long a, unsigned long long b,
                                                      unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long af_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long af_pair(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void af_unpair(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void af_cp16(float* smem, const float* gmem, bool ok) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(gmem),
               "r"(ok ? 16 : 0));
}

template <int D, int BM, int TM>
__global__ void __launch_bounds__(BM / TM * 16) attention_f32_kernel(
    const float* __restrict__ q, const float* __restrict__ k_cache,
    const float* __restrict__ v_cache, const int* __restrict__ q_start,
    const int* __restrict__ positions, const int* __restrict__ tables, int table_stride,
    float* __restrict__ out, int nh, int nkv, int page_size, int num_pages, int window,
    float scale_log2, int* __restrict__ err, int bufs) {
  constexpr int THREADS = BM / TM * 16, P = D + 4, PP = AF_KEYS + 4, CJ = D / 64;
  constexpr int CHUNKS = D / 4;                 // 16-byte pieces of a row
  extern __shared__ __align__(16) float af_smem[];
  float* Qs = af_smem;                          // [BM][P]
  float* Ks = Qs + BM * P;                      // [bufs][64][P]
  float* Vs = Ks + bufs * AF_KEYS * P;          // [bufs][64][P]
  float* Ps = Vs + bufs * AF_KEYS * P;          // [BM][PP]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int g = blockIdx.y, b = blockIdx.z, Gh = nh / nkv;
  const int t0 = q_start[b], n_tok = q_start[b + 1] - t0;
  // (the last rows see the most keys and start first)
  const int rows = n_tok * Gh, row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * BM;
  if (row0 >= rows) return;
  const int* table = tables + (size_t)b * table_stride;
  const int p_lo = positions[t0 + row0 / Gh];
  const int p_hi = positions[t0 + min(row0 + BM - 1, rows - 1) / Gh];
  const int j_lo = window > 0 ? max(0, p_lo - window + 1) : 0;
  const int tile_a = j_lo / AF_KEYS, tile_b = p_hi / AF_KEYS + 1;

  // A warp takes OWN rows of the tile: its lanes look one row each up in the table (a lookup and a division
  // per 16-byte piece took longer than the tile's products), then whole rows are copied.
  constexpr int OWN = AF_KEYS / (THREADS / 32), AT_ONCE = 32 / CHUNKS;
  static_assert(THREADS % 32 == 0 && OWN >= AT_ONCE && OWN <= 32, "rows of a warp");
  const int lane = tid & 31, own0 = tid / 32 * OWN;
  auto load = [&](int tile, int buf) {
    const int e = tile * AF_KEYS + own0 + lane;
    long long at = -1;
    if (lane < OWN && e >= j_lo && e <= p_hi) {
      const int lp = e / page_size, page = table[lp];
      if (page < 0 || page >= num_pages) atomicOr(err, BF_ERR_PAGE);
      else at = (((long long)page * nkv + g) * page_size + (e - lp * page_size)) * D;
    }
    const int c = lane % CHUNKS * 4;
#pragma unroll
    for (int i = 0; i < OWN; i += AT_ONCE) {
      const int r = i + lane / CHUNKS;
      const long long from = __shfl_sync(0xffffffffu, at, r);
      const bool ok = from >= 0;
      const size_t off = ok ? (size_t)(from + c) : 0;
      af_cp16(Ks + (buf * AF_KEYS + own0 + r) * P + c, k_cache + off, ok);
      af_cp16(Vs + (buf * AF_KEYS + own0 + r) * P + c, v_cache + off, ok);
    }
    cp_async_commit();
  };
  for (int i = tid; i < BM * CHUNKS; i += THREADS) {
    const int r = i / CHUNKS, c = i - r * CHUNKS, row = row0 + r;
    const bool ok = row < rows;
    const size_t at = ok ? (size_t)(t0 + row / Gh) * nh * D + (size_t)(g * Gh + row % Gh) * D + c * 4
                         : 0;
    af_cp16(Qs + r * P + c * 4, q + at, ok);
  }
  load(tile_a, 0);

  int pos[TM];
  float m[TM], l[TM];
  unsigned long long o[TM][CJ][2];
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = row0 + ty * TM + i;
    pos[i] = row < rows ? positions[t0 + row / Gh] : -1;
    m[i] = -FLT_MAX;      // (not -inf: a score may be that, and counts as none)
    l[i] = 0.f;
#pragma unroll
    for (int j = 0; j < CJ; ++j) o[i][j][0] = o[i][j][1] = 0ull;
  }
  for (int tile = tile_a; tile < tile_b; ++tile) {
    if (bufs == 1 && tile > tile_a) {           // (a context longer than the caller said)
      __syncthreads();
      load(tile, 0);
    }
    const int buf = bufs == 1 ? 0 : (tile - tile_a) & 1;
    cp_async_wait<0>();
    __syncthreads();                            // the tile is here; the other buffer is used up
    if (bufs == 2 && tile + 1 < tile_b) load(tile + 1, buf ^ 1);
    const float* Kt = Ks + buf * AF_KEYS * P;
    const float* Vt = Vs + buf * AF_KEYS * P;
    unsigned long long s2[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
#pragma unroll 8
    for (int d = 0; d < D; d += 4) {
      ulonglong2 a[TM], kk[4];
#pragma unroll
      for (int i = 0; i < TM; ++i)
        a[i] = *reinterpret_cast<const ulonglong2*>(Qs + (ty * TM + i) * P + d);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        kk[j] = *reinterpret_cast<const ulonglong2*>(Kt + (tx + 16 * j) * P + d);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s2[i][j] = af_fma2(a[i].x, kk[j].x, s2[i][j]);
          s2[i][j] = af_fma2(a[i].y, kk[j].y, s2[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int lo = window > 0 ? pos[i] - window + 1 : 0;
      float s[4], mx = -INFINITY;
      bool seen[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int e = tile * AF_KEYS + tx + 16 * j;
        float x, y;
        af_unpair(s2[i][j], x, y);
        s[j] = x + y;
        seen[j] = e <= pos[i] && e >= lo;
        if (seen[j]) mx = fmaxf(mx, s[j] * scale_log2);
      }
#pragma unroll
      for (int w = 1; w < 16; w <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
      const float m_new = fmaxf(m[i], mx);
      const float corr = m_new == m[i] ? 1.f : exp2f(m[i] - m_new);   // (the first one: 0)
      m[i] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = seen[j] ? exp2f(fmaf(s[j], scale_log2, -m_new)) : 0.f;
        sum += p;
        Ps[(ty * TM + i) * PP + tx + 16 * j] = p;
      }
#pragma unroll
      for (int w = 1; w < 16; w <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
      l[i] = fmaf(l[i], corr, sum);
      const unsigned long long c2 = af_pair(corr, corr);
#pragma unroll
      for (int j = 0; j < CJ; ++j) {
        o[i][j][0] = af_mul2(o[i][j][0], c2);
        o[i][j][1] = af_mul2(o[i][j][1], c2);
      }
    }
    // keys that are here and that some row does not see: behind the first row's position, before the
    // last row's window
    bool odd = false;
    if (p_lo < p_hi && ((tile + 1) * AF_KEYS - 1 > p_lo ||
                        (window > 0 && tile * AF_KEYS < p_hi - window + 1))) {
      for (int i = tid; i < AF_KEYS * CHUNKS; i += THREADS) {
        const float4 x = *reinterpret_cast<const float4*>(Vt + i / CHUNKS * P + i % CHUNKS * 4);
        // (a number times zero is zero if it is finite, and only then)
        odd |= !(x.x * 0.f + x.y * 0.f + x.z * 0.f + x.w * 0.f == 0.f);
      }
      odd = __syncthreads_or(odd);
    }
    __syncwarp();                               // a row's probabilities come from its own half warp
    if (odd) {
      for (int e = 0; e < AF_KEYS; ++e) {
        const int key = tile * AF_KEYS + e;
        ulonglong2 v[CJ];
#pragma unroll
        for (int j = 0; j < CJ; ++j)
          v[j] = *reinterpret_cast<const ulonglong2*>(Vt + e * P + 4 * tx + 64 * j);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          if (key > pos[i] || (window > 0 && key < pos[i] - window + 1)) continue;
          const float w = Ps[(ty * TM + i) * PP + e];
          const unsigned long long w2 = af_pair(w, w);
#pragma unroll
          for (int j = 0; j < CJ; ++j) {
            o[i][j][0] = af_fma2(w2, v[j].x, o[i][j][0]);
            o[i][j][1] = af_fma2(w2, v[j].y, o[i][j][1]);
          }
        }
      }
      continue;
    }
#pragma unroll 4
    for (int e = 0; e < AF_KEYS; e += 4) {
      float4 p[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i)
        p[i] = *reinterpret_cast<const float4*>(Ps + (ty * TM + i) * PP + e);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        ulonglong2 v[CJ];
#pragma unroll
        for (int j = 0; j < CJ; ++j)
          v[j] = *reinterpret_cast<const ulonglong2*>(Vt + (e + x) * P + 4 * tx + 64 * j);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float w = x == 0 ? p[i].x : x == 1 ? p[i].y : x == 2 ? p[i].z : p[i].w;
          const unsigned long long w2 = af_pair(w, w);
#pragma unroll
          for (int j = 0; j < CJ; ++j) {
            o[i][j][0] = af_fma2(w2, v[j].x, o[i][j][0]);
            o[i][j][1] = af_fma2(w2, v[j].y, o[i][j][1]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = row0 + ty * TM + i;
    if (row >= rows) continue;
    const float inv = 1.f / l[i];
    float* dst = out + (size_t)(t0 + row / Gh) * nh * D + (size_t)(g * Gh + row % Gh) * D + 4 * tx;
#pragma unroll
    for (int j = 0; j < CJ; ++j) {
      float4 r;
      af_unpair(o[i][j][0], r.x, r.y);
      af_unpair(o[i][j][1], r.z, r.w);
      *reinterpret_cast<float4*>(dst + 64 * j) =
          make_float4(r.x * inv, r.y * inv, r.z * inv, r.w * inv);
    }
  }
}

template <int D, int BM, int TM>
static int af_launch(const float* q, const float* k, const float* v, const int* q_start,
                     const int* positions, const int* tables, int table_stride, float* out, int B,
                     int max_q, int nh, int nkv, int page_size, int num_pages, int window,
                     float scale, int bufs, int* err, cudaStream_t stream) {
  const auto bytes = [](int n) {
    return ((size_t)BM * (D + 4) + (size_t)2 * n * AF_KEYS * (D + 4) +
            (size_t)BM * (AF_KEYS + 4)) * sizeof(float);
  };
  const size_t smem = bytes(bufs);
  auto kern = attention_f32_kernel<D, BM, TM>;
  static bool configured[BF_MAX_DEVICES];
  bool& done = configured[bf_current_device()];
  if (!done) {
    const cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(2));
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const long long rows = (long long)max_q * (nh / nkv);
  kern<<<dim3((unsigned)((rows + BM - 1) / BM), nkv, B), BM / TM * 16, smem, stream>>>(
      q, k, v, q_start, positions, tables, table_stride, out, nh, nkv, page_size, num_pages, window,
      scale * 1.4426950408889634f, err, bufs);
  return bf_launch_status();
}

// q and out [T, nh, d] contiguous; request b's token rows q_start[b] .. q_start[b + 1] - 1, at most
// max_q of them, its pages in tables[b]; window 0: every earlier key; max_ctx: the longest context, or
// 0 (contexts of one tile need one buffer for K and V, and three CTAs of four rows fit an SM instead of
// one: 48 single tokens of 8 kv heads of 128 behind 0 and 15 keys 17 and 20 us -> 8.4 and 9.8, then with the
// rows' lookups 7.6 and 7.7; the kernel for any size 7.9 and 18.5).
BF_EXPORT int bf_attention_f32(const float* q, const float* k_cache, const float* v_cache,
                               const int* q_start, const int* positions, const int* tables,
                               int table_stride, float* out, int B, int max_q, int nh, int nkv,
                               int d, int page_size, int num_pages, int window, float scale,
                               int max_ctx, int* err, cudaStream_t stream) {
  if (B <= 0 || max_q <= 0) return 0;
  if (nkv <= 0 || nh % nkv || nkv > 65535 || B > 65535 || (d != 64 && d != 128) || !(scale > 0.f) ||
      (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15))
    return (int)cudaErrorInvalidValue;
  // few rows from every request of the step (single tokens alone): tiles of four, each with as many
  // threads a row, so that the chain from key tile to key tile is short
  const int bufs = max_ctx > 0 && max_ctx <= AF_KEYS ? 1 : 2;
  const long long rows = (long long)max_q * (nh / nkv);
  const bool few = rows <= 16;
  // tiles of 64 rows, or of 32 where those would leave SMs idle: a key tile of half the rows takes half
  // the time, and the CTA of the last rows, which walks them all, is what a short portion waits for (333
  // tokens of 16 heads, 8 kv heads of 128: 60 -> 38 us with the rows' lookups; threads of two rows
  // instead of four 45)
  const bool small = (rows + 63) / 64 * nkv * B < 148;
#define AF_GO(D)                                                                                \
  (few ? af_launch<D, 4, 1>(q, k_cache, v_cache, q_start, positions, tables, table_stride, out, \
                            B, max_q, nh, nkv, page_size, num_pages, window, scale, bufs, err, stream) \
   : small ? af_launch<D, 32, 4>(q, k_cache, v_cache, q_start, positions, tables, table_stride, out, B, max_q, \
                                 nh, nkv, page_size, num_pages, window, scale, bufs, err, stream) \
       : af_launch<D, 64, 4>(q, k_cache, v_cache, q_start, positions, tables, table_stride, out, \
                             B, max_q, nh, nkv, page_size, num_pages, window, scale, bufs, err, stream))
  return d == 64 ? AF_GO(64) : AF_GO(128);
#undef AF_GO
}
