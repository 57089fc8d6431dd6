// Recurrences over a matrix state in chunks of tokens, for the bfloat16 engine's prompt portions:
// what retention.cu (linear scan) and mlstm.cu (matrix memory) walk token by token, as products.
//
//   linear:  S_t = d_t S_{t-1} + k_t v_t^T                        o_t = S_t^T q_t
//   mLSTM:   the same with d_t = exp(f_t + m_{t-1} - m_t), k_t v_t^T times exp(i_t - m_t), a vector
//            n_t beside S_t that takes k_t alone, and o_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6)
//
// With F_t the sum of the log decays up to token t, H_s = F_s - i_s and G_t = min(-m_0, min_{s <= t}
// H_s) (linear: i = m = 0 and G = H = F), token s reaches token t with the weight exp(G_t - H_s)
// <= 1 and the state before a chunk whose last earlier token is c with exp(G_t - G_c); for the
// mLSTM m_t = F_t - G_t.  F, G and H are double, so a difference of two of them is good to a
// float's last bit; every product below is float (FP32 multiply-adds, no tensor-core mode), every
// sum of one order.  Per chunk of `C` tokens and head:
//
//   cs_gates   F, G, H of every token; one block per (head, request)
//   cs_qk      Q K^T of a chunk, once per q/k head (several heads may share them)
//   cs_state   U = sum_s exp(G_last - H_s) k_s v_s^T: what the chunk adds to the state
//   cs_prefix  from chunk to chunk: S <- exp(G_last - G_c) S + U; U's place takes the state before
//              the chunk; the request's slot takes the last one
//   cs_out     o = [exp(G_t - G_c) q_t | exp(G_t - H_s) (q_t . k_s)] [S ; V]: one product with dk +
//              C terms, the weights applied as its operands are stored into shared memory
//
// Measured (GPU time of the kernels / of the walk): 2,000 tokens, 64 heads of 128 x 64 over 8
// q/k heads: 220 / 459 us (cs_out 96, cs_state 76, cs_prefix 23, cs_qk 14, cs_gates 11); 2,048 tokens
// of 8 heads of 128 x 256: 127 / 289; mLSTM, 8 heads of 256 x 512: 394 / 979 (168, 138, 54, 22, 12).
// Error against 64 bits, decays of 0.98 to 1: o 1.4e-7 (walk 1.9e-7), state 1.1e-7 (1.8e-7); mLSTM: o
// 5e-6 (2e-5), state 0.9e-7 (4.0e-7).
//
// Why: the walk has heads x dk x dv independent elements and a chain of multiply-adds from token to
// token, so it left the FP32 pipes at 15 to 20 % (see those files); the products have no chain and
// reach what the float32 product of sgemm_f32.cu reaches.  They are built like it: 64 x 64 outputs
// a CTA, 16 terms a step fetched a step ahead, packed multiply-adds of row pairs.
//
// Requests of at most `n_min` tokens have no chunks here (the walk serves them).  The order of sums
// depends on where a step's portions begin, so the float32 engine, whose results must not depend
// on the cut, does not use these kernels.
#include "common.cuh"

#define CS_THREADS 128
#define CS_T 64            // tile edge
#define CS_K 16            // terms a step
#define CS_P (CS_T + 4)    // pitch of a staged row of 64

__device__ __forceinline__ unsigned long long cs_pair(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void cs_unpair(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long cs_fma2(unsigned long long a, unsigned long long b,
                                                      unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long cs_add2(unsigned long long a,
                                                      unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ float4 cs_ld4(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ float4 cs_ld4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 cs_zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float4 cs_times(float4 v, float f) {
  return make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
}

// ------------------------------------------------------------------------ which chunk is it
struct CsChunk {
  int b;        // request, -1: no such chunk
  int first;    // the request's first chunk
  int index;    // the chunk's number inside the request
  int t0;       // the request's first token
  int n;        // the request's tokens
};

// Chunk `id` of all requests' chunks in order, or (want_b >= 0) request want_b's first chunk.
// Called by whole warps.
__device__ __forceinline__ CsChunk cs_find(const int* __restrict__ q_start, int B, int C,
                                           int n_min, int id, int want_b) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int b0 = 0; b0 < B; b0 += 32) {
    const int b = b0 + lane;
    int t0 = 0, n = 0;
    if (b < B) {
      t0 = q_start[b];
      n = q_start[b + 1] - t0;
    }
    const int own = n > n_min ? (n + C - 1) / C : 0;
    int sum = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    const int mine = before + sum - own;           // this lane's first chunk
    const bool hit = want_b >= 0 ? b == want_b && b < B : id >= mine && id < mine + own;
    const unsigned vote = __ballot_sync(0xffffffffu, hit);
    if (vote) {
      const int src = __ffs(vote) - 1;
      CsChunk c;
      c.b = b0 + src;
      c.first = __shfl_sync(0xffffffffu, mine, src);
      c.t0 = __shfl_sync(0xffffffffu, t0, src);
      c.n = __shfl_sync(0xffffffffu, n, src);
      c.index = want_b >= 0 ? 0 : id - c.first;
      return c;
    }
    before += __shfl_sync(0xffffffffu, sum, 31);
  }
  CsChunk none = {-1, 0, 0, 0, 0};
  return none;
}

// ------------------------------------------------------------------------------- cs_gates
#define CS_GATE_THREADS 256

__device__ __forceinline__ double cs_log_decay(float d) {
  // a decay that underflowed to zero forgets everything: exp(-1e4) is zero in float
  return d > 0.f ? fmax(log((double)d), -1e4) : -1e4;
}

// Exclusive scan over the block's threads of `v` by + or min; `seed` comes before the first.
template <bool MIN>
__device__ __forceinline__ double cs_block_scan(double v, double seed, double* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x = MIN ? fmin(x, y) : x + y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  double base = seed;
  for (int w = 0; w < warp; ++w) base = MIN ? fmin(base, sh[w]) : base + sh[w];
  const double prev = __shfl_up_sync(0xffffffffu, x, 1);
  __syncthreads();
  if (lane == 0) return base;
  return MIN ? fmin(base, prev) : base + prev;
}

// G and Hs [H][T]; mLSTM: E [H][T] = exp(-m_t), and the slot's m becomes the last token's
// (g0 [B][H] keeps minus the earlier one for the kernels behind).
template <bool MLSTM>
__global__ void __launch_bounds__(CS_GATE_THREADS) cs_gates_kernel(
    const float* __restrict__ decays, const float* __restrict__ tok_decay,
    const float* __restrict__ gates, float* __restrict__ state, long long slot_stride,
    int state_size, const int* __restrict__ q_start, const int* __restrict__ state_slots,
    int n_slots, double* __restrict__ G, double* __restrict__ Hs, float* __restrict__ E,
    double* __restrict__ g0, int T, int H, int dkdv, int dk, int n_min) {
  __shared__ double sh[CS_GATE_THREADS / 32];
  const int h = blockIdx.x, b = blockIdx.y;
  const int t0 = q_start[b], n = q_start[b + 1] - t0;
  if (n <= n_min) return;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= n_slots) return;         // (flagged by cs_prefix)
  const int per = (n + CS_GATE_THREADS - 1) / CS_GATE_THREADS;
  const int a = min(n, (int)threadIdx.x * per), e = min(n, a + per);
  double* g = G + (size_t)h * T + t0;
  double* hs = Hs + (size_t)h * T + t0;
  const double fixed = MLSTM || tok_decay ? 0.0 : cs_log_decay(decays[h]);
  auto log_decay = [&](int t) -> double {
    if (MLSTM) return (double)gates[(size_t)(t0 + t) * 2 * H + H + h];
    return tok_decay ? cs_log_decay(tok_decay[(size_t)(t0 + t) * H + h]) : fixed;
  };
  double F = 0.0;
  for (int t = a; t < e; ++t) {
    F += log_decay(t);
    hs[t] = F;
  }
  const double off = cs_block_scan<false>(F, 0.0, sh);
  if (!MLSTM) {
    for (int t = a; t < e; ++t) {
      const double x = hs[t] + off;
      hs[t] = x;
      g[t] = x;
    }
    if (threadIdx.x == 0) g0[(size_t)b * H + h] = 0.0;
    return;
  }
  double low = 1e300;
  for (int t = a; t < e; ++t)
    low = fmin(low, hs[t] + off - (double)gates[(size_t)(t0 + t) * 2 * H + h]);
  float* m_at = state + (size_t)slot * slot_stride + (size_t)h * state_size + dkdv + dk;
  const double m0 = (double)*m_at;
  double run = cs_block_scan<true>(low, -m0, sh);  // (its barriers order this read before the write)
  for (int t = a; t < e; ++t) {
    const double x = hs[t] + off;
    const double hv = x - (double)gates[(size_t)(t0 + t) * 2 * H + h];
    run = fmin(run, hv);
    hs[t] = hv;
    g[t] = run;
    E[(size_t)h * T + t0 + t] = expf((float)(run - x));
    if (t == n - 1) *m_at = (float)(x - run);
  }
  if (threadIdx.x == 0) g0[(size_t)b * H + h] = -m0;
}

// ---------------------------------------------------------------------- the products' tiles
// 64 x 64 outputs of a CTA of 128 threads: thread (tx, ty) has rows 8 ty .. 8 ty + 7 (four pairs)
// and columns 4 tx .. 4 tx + 3.  A step's sixteen terms are summed on their own and then added: a
// sum's rounding grows with the square root of 16 + terms / 16, not of the terms (o of 2,000 tokens
// with decays spread over 0 .. 1 was 2.1e-7 from 64 bits with one chain, the walk 0.8e-7).
typedef unsigned long long CsAcc[4][4];

__device__ __forceinline__ void cs_clear(CsAcc& acc) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
}

__device__ __forceinline__ void cs_mul(const float (&As)[CS_K][CS_P], const float (&Bs)[CS_K][CS_P],
                                       int tx, int ty, CsAcc& total) {
  CsAcc acc;
  cs_clear(acc);
#pragma unroll
  for (int kk = 0; kk < CS_K; ++kk) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(&As[kk][ty * 8]);
    const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(&As[kk][ty * 8 + 4]);
    const float4 w = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
    const unsigned long long a[4] = {a0.x, a0.y, a1.x, a1.y};
    const unsigned long long b[4] = {cs_pair(w.x, w.x), cs_pair(w.y, w.y), cs_pair(w.z, w.z),
                                     cs_pair(w.w, w.w)};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = cs_fma2(a[i], b[j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) total[i][j] = cs_add2(total[i][j], acc[i][j]);
}

// A step's pieces of four: `idx` 0..255, two a thread.  Rows with the terms side by side (row
// idx / 4, terms 4 (idx % 4) ..) are turned on their way into shared memory; rows of terms (term
// idx / 16, columns 4 (idx % 16) ..) go in as they are.
__device__ __forceinline__ void cs_put_turned(float (&S)[CS_K][CS_P], int idx, float4 v) {
  const int r = idx >> 2, k = (idx & 3) * 4;
  S[k][r] = v.x;
  S[k + 1][r] = v.y;
  S[k + 2][r] = v.z;
  S[k + 3][r] = v.w;
}
__device__ __forceinline__ void cs_put(float (&S)[CS_K][CS_P], int idx, float4 v) {
  *reinterpret_cast<float4*>(&S[idx >> 4][(idx & 15) * 4]) = v;
}

struct CsIn {
  long long q_off, k_off, v_off;      // of head 0, in elements of a token's row
  long long qk_stride, v_stride;      // from token to token
  int H, QH, dk, dv, C, T, B, n_min;
  float q_scale;
};

// ---------------------------------------------------------------------------------- cs_qk
// grid (chunks, QH, row tiles x column tiles): qkm[chunk][qh][C][C], the tiles at and below the
// diagonal
template <typename A>
__global__ void __launch_bounds__(CS_THREADS) cs_qk_kernel(
    const A* __restrict__ qk, CsIn p, const int* __restrict__ q_start, float* __restrict__ qkm) {
  __shared__ __align__(16) float As[2][CS_K][CS_P], Bs[2][CS_K][CS_P];
  const int tiles = p.C / CS_T;
  const int rt = blockIdx.z / tiles, ct = blockIdx.z % tiles;
  if (ct > rt) return;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, blockIdx.x, -1);
  if (c.b < 0) return;
  const int at = c.index * p.C;                  // the chunk's first token inside the request
  const int n = min(p.C, c.n - at);
  if (rt * CS_T >= n) return;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int hq = blockIdx.y;
  const A* q = qk + (size_t)(c.t0 + at) * p.qk_stride + p.q_off + (size_t)hq * p.dk;
  const A* k = qk + (size_t)(c.t0 + at) * p.qk_stride + p.k_off + (size_t)hq * p.dk;
  CsAcc acc;
  cs_clear(acc);
  float4 fa[2], fb[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int idx = tid + x * CS_THREADS, r = idx >> 2, kk = k0 + (idx & 3) * 4;
      const int ra = rt * CS_T + r, rb = ct * CS_T + r;
      fa[x] = ra < n && kk < p.dk ? cs_ld4(q + (size_t)ra * p.qk_stride + kk) : cs_zero();
      fb[x] = rb < n && kk < p.dk ? cs_ld4(k + (size_t)rb * p.qk_stride + kk) : cs_zero();
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      cs_put_turned(As[buf], tid + x * CS_THREADS, fa[x]);
      cs_put_turned(Bs[buf], tid + x * CS_THREADS, fb[x]);
    }
  };
  fetch(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < p.dk; k0 += CS_K, buf ^= 1) {
    if (k0 + CS_K < p.dk) fetch(k0 + CS_K);
    cs_mul(As[buf], Bs[buf], tx, ty, acc);
    if (k0 + CS_K < p.dk) store(buf ^ 1);
    __syncthreads();
  }
  float* dst = qkm + ((size_t)blockIdx.x * p.QH + hq) * p.C * p.C;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) cs_unpair(acc[i][j], lo[j], hi[j]);
    const int r = rt * CS_T + ty * 8 + 2 * i, col = ct * CS_T + tx * 4;
    const float f = p.q_scale;
    *reinterpret_cast<float4*>(dst + (size_t)r * p.C + col) =
        make_float4(lo[0] * f, lo[1] * f, lo[2] * f, lo[3] * f);
    *reinterpret_cast<float4*>(dst + (size_t)(r + 1) * p.C + col) =
        make_float4(hi[0] * f, hi[1] * f, hi[2] * f, hi[3] * f);
  }
}

// ------------------------------------------------------------------------------- cs_state
// grid (chunks, H, row tiles x column tiles).  U[chunk][h]: linear [dv][dk], mLSTM [dk][dv] (each
// like its state); mLSTM: Un[chunk][h][dk] by the CTAs of the first column tile.
template <typename A, typename V, bool MLSTM>
__global__ void __launch_bounds__(CS_THREADS) cs_state_kernel(
    const A* __restrict__ qk, const V* __restrict__ vsrc, CsIn p, const int* __restrict__ q_start,
    const double* __restrict__ G, const double* __restrict__ Hs, float* __restrict__ U,
    float* __restrict__ Un) {
  __shared__ __align__(16) float As[2][CS_K][CS_P], Bs[2][CS_K][CS_P];
  __shared__ float ws[2][CS_K];
  const int rows = MLSTM ? p.dk : p.dv, cols = MLSTM ? p.dv : p.dk;
  const int cts = (cols + CS_T - 1) / CS_T;
  const int r0 = (blockIdx.z / cts) * CS_T, c0 = (blockIdx.z % cts) * CS_T;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, blockIdx.x, -1);
  if (c.b < 0) return;
  const int at = c.index * p.C;
  const int n = min(p.C, c.n - at);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int h = blockIdx.y, hq = h / (p.H / p.QH);
  const A* k = qk + (size_t)(c.t0 + at) * p.qk_stride + p.k_off + (size_t)hq * p.dk;
  const V* v = vsrc + (size_t)(c.t0 + at) * p.v_stride + p.v_off + (size_t)h * p.dv;
  const double* hs = Hs + (size_t)h * p.T + c.t0 + at;
  const double g_last = G[(size_t)h * p.T + c.t0 + at + n - 1];
  CsAcc acc;
  cs_clear(acc);
  float nacc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) nacc[i] = 0.f;
  float4 fk[2], fv[2];
  float fw[2];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int idx = tid + x * CS_THREADS, s = s0 + (idx >> 4), d = (idx & 15) * 4;
      const int dkk = (MLSTM ? r0 : c0) + d, dvv = (MLSTM ? c0 : r0) + d;
      fw[x] = s < n ? expf((float)(g_last - hs[s])) : 0.f;
      fk[x] = s < n && dkk < p.dk ? cs_ld4(k + (size_t)s * p.qk_stride + dkk) : cs_zero();
      fv[x] = s < n && dvv < p.dv ? cs_ld4(v + (size_t)s * p.v_stride + dvv) : cs_zero();
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int idx = tid + x * CS_THREADS;
      cs_put(MLSTM ? As[buf] : Bs[buf], idx, fk[x]);
      cs_put(MLSTM ? Bs[buf] : As[buf], idx, cs_times(fv[x], fw[x]));
      if (MLSTM && (idx & 15) == 0) ws[buf][idx >> 4] = fw[x];
    }
  };
  fetch(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int s0 = 0; s0 < n; s0 += CS_K, buf ^= 1) {
    if (s0 + CS_K < n) fetch(s0 + CS_K);
    cs_mul(As[buf], Bs[buf], tx, ty, acc);
    if (MLSTM && c0 == 0) {
      // n's share: term tx of the step's sixteen, for this thread's eight rows
      const float w = ws[buf][tx];
#pragma unroll
      for (int i = 0; i < 8; ++i) nacc[i] = fmaf(As[buf][tx][ty * 8 + i], w, nacc[i]);
    }
    if (s0 + CS_K < n) store(buf ^ 1);
    __syncthreads();
  }
  float* dst = U + ((size_t)blockIdx.x * p.H + h) * p.dk * p.dv;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) cs_unpair(acc[i][j], lo[j], hi[j]);
    const int r = r0 + ty * 8 + 2 * i, col = c0 + tx * 4;
    if (col < cols) {
      if (r < rows)
        *reinterpret_cast<float4*>(dst + (size_t)r * cols + col) =
            make_float4(lo[0], lo[1], lo[2], lo[3]);
      if (r + 1 < rows)
        *reinterpret_cast<float4*>(dst + (size_t)(r + 1) * cols + col) =
            make_float4(hi[0], hi[1], hi[2], hi[3]);
    }
  }
  if (MLSTM && c0 == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) nacc[i] += __shfl_xor_sync(0xffffffffu, nacc[i], o);
      const int r = r0 + ty * 8 + i;
      if (tx == 0 && r < p.dk) Un[((size_t)blockIdx.x * p.H + h) * p.dk + r] = nacc[i];
    }
  }
}

// ------------------------------------------------------------------------------- cs_prefix
// grid (pieces of 4 x 128 state elements (mLSTM: n behind them), H, B)
#define CS_AHEAD 4
template <bool MLSTM>
__global__ void __launch_bounds__(128) cs_prefix_kernel(
    float* __restrict__ state, long long slot_stride, int state_size,
    const int* __restrict__ state_slots, int n_slots, CsIn p, const int* __restrict__ q_start,
    const double* __restrict__ G, const double* __restrict__ g0, float* __restrict__ U,
    float* __restrict__ Un, int* __restrict__ err) {
  const int h = blockIdx.y, b = blockIdx.z;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, 0, b);
  if (c.n <= p.n_min) return;
  const int slot = state_slots[b];
  if (slot < 0 || slot >= n_slots) {
    if (threadIdx.x == 0) atomicOr(err, BF_ERR_SLOT);
    return;
  }
  const int size = p.dk * p.dv;
  const int e = (blockIdx.x * 128 + threadIdx.x) * 4;
  float* s_at = state + (size_t)slot * slot_stride + (size_t)h * state_size + e;
  float* u = U + ((size_t)c.first * p.H + h) * size + e;
  size_t step = (size_t)p.H * size;
  if (e >= size) {
    if (!MLSTM || e - size >= p.dk) return;
    u = Un + ((size_t)c.first * p.H + h) * p.dk + (e - size);
    step = (size_t)p.H * p.dk;
  }
  const int chunks = (c.n + p.C - 1) / p.C;
  const double* g = G + (size_t)h * p.T + c.t0;
  double before = g0[(size_t)b * p.H + h];
  float4 S = *reinterpret_cast<const float4*>(s_at);
  float4 next[CS_AHEAD];
#pragma unroll
  for (int i = 0; i < CS_AHEAD; ++i)
    if (i < chunks) next[i] = *reinterpret_cast<const float4*>(u + i * step);
  for (int i0 = 0; i0 < chunks; i0 += CS_AHEAD) {
#pragma unroll
    for (int j = 0; j < CS_AHEAD; ++j) {
      const int i = i0 + j;
      if (i < chunks) {
        const float4 add = next[j];
        if (i + CS_AHEAD < chunks)
          next[j] = *reinterpret_cast<const float4*>(u + (size_t)(i + CS_AHEAD) * step);
        *reinterpret_cast<float4*>(u + (size_t)i * step) = S;
        const double last = g[min(c.n, (i + 1) * p.C) - 1];
        const float d = expf((float)(last - before));
        before = last;
        S = make_float4(fmaf(d, S.x, add.x), fmaf(d, S.y, add.y), fmaf(d, S.z, add.z),
                        fmaf(d, S.w, add.w));
      }
    }
  }
  *reinterpret_cast<float4*>(s_at) = S;
}

// ---------------------------------------------------------------------------------- cs_out
// grid (chunks, H, row tiles x column tiles of dv)
template <typename A, typename V, bool MLSTM>
__global__ void __launch_bounds__(CS_THREADS) cs_out_kernel(
    const A* __restrict__ qk, const V* __restrict__ vsrc, CsIn p, const int* __restrict__ q_start,
    const int* __restrict__ state_slots, int n_slots, const double* __restrict__ G,
    const double* __restrict__ Hs, const double* __restrict__ g0, const float* __restrict__ E,
    const float* __restrict__ qkm, const float* __restrict__ U, const float* __restrict__ Un,
    float* __restrict__ o_raw) {
  __shared__ __align__(16) float As[2][CS_K][CS_P], Bs[2][CS_K][CS_P];
  __shared__ double gt[CS_T];
  __shared__ float at_s[CS_T], ns[2][CS_K];
  const int cts = (p.dv + CS_T - 1) / CS_T;
  const int rt = blockIdx.z / cts, c0 = (blockIdx.z % cts) * CS_T;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, blockIdx.x, -1);
  if (c.b < 0) return;
  const int slot = state_slots[c.b];
  if (slot < 0 || slot >= n_slots) return;
  const int at = c.index * p.C;
  const int n = min(p.C, c.n - at);
  const int r0 = rt * CS_T;
  if (r0 >= n) return;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int h = blockIdx.y, hq = h / (p.H / p.QH);
  const A* q = qk + (size_t)(c.t0 + at) * p.qk_stride + p.q_off + (size_t)hq * p.dk;
  const V* v = vsrc + (size_t)(c.t0 + at) * p.v_stride + p.v_off + (size_t)h * p.dv;
  const double* g = G + (size_t)h * p.T + c.t0 + at;
  const double* hs = Hs + (size_t)h * p.T + c.t0 + at;
  const double before = c.index ? g[-1] : g0[(size_t)c.b * p.H + h];
  const float* P = qkm + ((size_t)blockIdx.x * p.QH + hq) * p.C * p.C + (size_t)r0 * p.C;
  const float* S = U + ((size_t)blockIdx.x * p.H + h) * p.dk * p.dv;
  const float* nst = Un + ((size_t)blockIdx.x * p.H + h) * p.dk;
  if (tid < CS_T) {
    const double x = r0 + tid < n ? g[r0 + tid] : 0.0;
    gt[tid] = x;
    at_s[tid] = r0 + tid < n ? expf((float)(x - before)) * p.q_scale : 0.f;
  }
  __syncthreads();
  CsAcc acc;
  cs_clear(acc);
  float den[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) den[i] = 0.f;
  // the terms: sizes 0 .. dk - 1 of q against the state, then tokens 0 .. s_end - 1 against v
  const int dk_pad = (p.dk + CS_K - 1) / CS_K * CS_K;
  const int s_end = min(n, r0 + CS_T);
  const int terms = dk_pad + s_end;
  float4 fa[2], fb[2];
  double fh[4];
  float fn = 0.f;
  auto fetch = [&](int k0) {
    if (k0 < dk_pad) {
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int idx = tid + x * CS_THREADS, r = idx >> 2, kk = k0 + (idx & 3) * 4;
        fa[x] = r0 + r < n && kk < p.dk ? cs_ld4(q + (size_t)(r0 + r) * p.qk_stride + kk)
                                        : cs_zero();
        if (MLSTM) {                           // S [dk][dv]: rows of terms
          const int kr = k0 + (idx >> 4), j = c0 + (idx & 15) * 4;
          fb[x] = kr < p.dk && j < p.dv ? cs_ld4(S + (size_t)kr * p.dv + j) : cs_zero();
        } else {                               // S [dv][dk]: rows with the terms side by side
          fb[x] = c0 + r < p.dv && kk < p.dk ? cs_ld4(S + (size_t)(c0 + r) * p.dk + kk)
                                             : cs_zero();
        }
      }
      if (MLSTM && tid < CS_K) fn = k0 + tid < p.dk ? nst[k0 + tid] : 0.f;
    } else {
      const int s0 = k0 - dk_pad;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int idx = tid + x * CS_THREADS;
        const int r = idx >> 2, s = s0 + (idx & 3) * 4;
        fa[x] = cs_ld4(P + (size_t)r * p.C + s);
        const int sv = s0 + (idx >> 4), j = c0 + (idx & 15) * 4;
        fb[x] = sv < n && j < p.dv ? cs_ld4(v + (size_t)sv * p.v_stride + j) : cs_zero();
      }
      const int s = s0 + (tid & 3) * 4;        // (both pieces of a thread have the same tokens)
#pragma unroll
      for (int y = 0; y < 4; ++y) fh[y] = s + y < n ? hs[s + y] : 0.0;
      fn = 1.f;
    }
  };
  auto store = [&](int buf, int k0) {
    if (k0 < dk_pad) {
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int idx = tid + x * CS_THREADS;
        cs_put_turned(As[buf], idx, cs_times(fa[x], at_s[idx >> 2]));
        if (MLSTM) cs_put(Bs[buf], idx, fb[x]);
        else cs_put_turned(Bs[buf], idx, fb[x]);
      }
    } else {
      const int s = k0 - dk_pad + (tid & 3) * 4;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int idx = tid + x * CS_THREADS, r = idx >> 2;
        // row r0 + r sees the chunk's tokens up to itself
        const double gr = gt[r];
        const int last = r0 + r < n ? r0 + r : -1;
        float4 w;
        w.x = s <= last ? fa[x].x * expf((float)(gr - fh[0])) : 0.f;
        w.y = s + 1 <= last ? fa[x].y * expf((float)(gr - fh[1])) : 0.f;
        w.z = s + 2 <= last ? fa[x].z * expf((float)(gr - fh[2])) : 0.f;
        w.w = s + 3 <= last ? fa[x].w * expf((float)(gr - fh[3])) : 0.f;
        cs_put_turned(As[buf], idx, w);
        cs_put(Bs[buf], idx, fb[x]);
      }
    }
    if (MLSTM && tid < CS_K) ns[buf][tid] = fn;
  };
  fetch(0);
  store(0, 0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < terms; k0 += CS_K, buf ^= 1) {
    if (k0 + CS_K < terms) fetch(k0 + CS_K);
    cs_mul(As[buf], Bs[buf], tx, ty, acc);
    if (MLSTM) {
      // n_t . q_t: the same rows against n and against ones; term tx of the step's sixteen
      const float w = ns[buf][tx];
#pragma unroll
      for (int i = 0; i < 8; ++i) den[i] = fmaf(As[buf][tx][ty * 8 + i], w, den[i]);
    }
    if (k0 + CS_K < terms) store(buf ^ 1, k0 + CS_K);
    __syncthreads();
  }
  if (MLSTM) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) den[i] += __shfl_xor_sync(0xffffffffu, den[i], o);
      const int r = r0 + ty * 8 + i;
      den[i] = r < n ? fmaxf(fabsf(den[i]), E[(size_t)h * p.T + c.t0 + at + r]) + 1e-6f : 1.f;
    }
  }
  const int col = c0 + tx * 4;
  if (col >= p.dv) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      cs_unpair(acc[i][j], lo[j], hi[j]);
      if (MLSTM) {
        lo[j] /= den[2 * i];
        hi[j] /= den[2 * i + 1];
      }
    }
    const int r = r0 + ty * 8 + 2 * i;
    float* dst = o_raw + ((size_t)(c.t0 + at + r) * p.H + h) * p.dv + col;
    if (r < n) *reinterpret_cast<float4*>(dst) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    if (r + 1 < n)
      *reinterpret_cast<float4*>(dst + (size_t)p.H * p.dv) = make_float4(hi[0], hi[1], hi[2], hi[3]);
  }
}

// -------------------------------------------------------------------------------- launches
// Scratch (bytes, each part on a 256-byte boundary): G, Hs, g0 | E (mLSTM) | qkm | U | Un (mLSTM).
struct CsLayout {
  size_t G, Hs, g0, E, qkm, U, Un, total;
  int chunks;
};
static CsLayout cs_layout(int T, int B, int H, int QH, int dk, int dv, int C, int mlstm) {
  CsLayout l;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 255) & ~(size_t)255;
    return here;
  };
  l.chunks = T / C + B;                // the most that portions of T tokens in all can have
  l.G = take((size_t)T * H * 8);
  l.Hs = take((size_t)T * H * 8);
  l.g0 = take((size_t)B * H * 8);
  l.E = take(mlstm ? (size_t)T * H * 4 : 0);
  l.qkm = take((size_t)l.chunks * QH * C * C * 4);
  l.U = take((size_t)l.chunks * H * dk * dv * 4);
  l.Un = take(mlstm ? (size_t)l.chunks * H * dk * 4 : 0);
  l.total = at;
  return l;
}

BF_EXPORT long long bf_chunk_scan_scratch(int T, int B, int H, int QH, int dk, int dv, int C,
                                          int mlstm) {
  return (long long)cs_layout(T, B, H, QH, dk, dv, C, mlstm).total;
}

template <typename A, typename V, bool MLSTM>
static int cs_launch(const A* qk, const V* v, const CsIn& p, const float* decays,
                     const float* tok_decay, const float* gates, float* state,
                     long long slot_stride, int state_size, const int* q_start,
                     const int* state_slots, int n_slots, float* o_raw, char* scratch, int* err,
                     cudaStream_t stream) {
  const CsLayout l = cs_layout(p.T, p.B, p.H, p.QH, p.dk, p.dv, p.C, MLSTM);
  double* G = (double*)(scratch + l.G);
  double* Hs = (double*)(scratch + l.Hs);
  double* g0 = (double*)(scratch + l.g0);
  float* E = (float*)(scratch + l.E);
  float* qkm = (float*)(scratch + l.qkm);
  float* U = (float*)(scratch + l.U);
  float* Un = (float*)(scratch + l.Un);
  const int tiles = p.C / CS_T, tk = (p.dk + CS_T - 1) / CS_T, tv = (p.dv + CS_T - 1) / CS_T;
  cs_gates_kernel<MLSTM><<<dim3(p.H, p.B), CS_GATE_THREADS, 0, stream>>>(
      decays, tok_decay, gates, state, slot_stride, state_size, q_start, state_slots, n_slots, G,
      Hs, E, g0, p.T, p.H, p.dk * p.dv, p.dk, p.n_min);
  cs_qk_kernel<A><<<dim3(l.chunks, p.QH, tiles * tiles), CS_THREADS, 0, stream>>>(qk, p, q_start,
                                                                                 qkm);
  cs_state_kernel<A, V, MLSTM><<<dim3(l.chunks, p.H, tk * tv), CS_THREADS, 0, stream>>>(
      qk, v, p, q_start, G, Hs, U, Un);
  const int elems = p.dk * p.dv + (MLSTM ? p.dk : 0);
  cs_prefix_kernel<MLSTM><<<dim3((elems + 511) / 512, p.H, p.B), 128, 0, stream>>>(
      state, slot_stride, state_size, state_slots, n_slots, p, q_start, G, g0, U, Un, err);
  cs_out_kernel<A, V, MLSTM><<<dim3(l.chunks, p.H, tiles * tv), CS_THREADS, 0, stream>>>(
      qk, v, p, q_start, state_slots, n_slots, G, Hs, g0, E, qkm, U, Un, o_raw);
  return bf_launch_status();
}

static bool cs_sizes_ok(const CsIn& p, const void* state, long long slot_stride) {
  return p.T > 0 && p.B > 0 && p.B <= 65535 && p.H > 0 && p.H <= 65535 && p.QH > 0 &&
         p.H % p.QH == 0 && p.dk > 0 && p.dv > 0 && p.dk % 4 == 0 && p.dv % 4 == 0 && p.C > 0 &&
         p.C % CS_T == 0 && p.qk_stride % 4 == 0 && p.v_stride % 4 == 0 && slot_stride % 4 == 0 &&
         ((uintptr_t)state & 15) == 0;
}

// qk [T][2][QH][dk] (q, then k), vf [T][H][dv], float; a decay per head or per (token, head).
// State and o_raw as in bf_linear_scan; requests of at most n_min tokens are left alone.
BF_EXPORT int bf_chunk_scan_linear(const float* qk, const float* vf, const float* decays,
                                   const float* tok_decay, float* state, long long slot_stride,
                                   const int* q_start, const int* state_slots, int n_slots,
                                   float* o_raw, void* scratch, int T, int B, int H, int QH,
                                   int dk, int dv, int C, int n_min, int* err,
                                   cudaStream_t stream) {
  CsIn p = {0, (long long)QH * dk, 0, 2LL * QH * dk, (long long)H * dv, H, QH, dk, dv, C, T, B,
            n_min, 1.f};
  if (!cs_sizes_ok(p, state, slot_stride) || (!decays && !tok_decay) || !scratch)
    return (int)cudaErrorInvalidValue;
  return cs_launch<float, float, false>(qk, vf, p, decays, tok_decay, nullptr, state, slot_stride,
                                        dk * dv, q_start, state_slots, n_slots, o_raw,
                                        (char*)scratch, err, stream);
}

// proj rows [q: H dk | k: H dk | v: H dv | ...] in bfloat16, gates and state as in bf_mlstm_scan.
BF_EXPORT int bf_chunk_scan_mlstm(const void* proj, long long stride, const float* gates,
                                  float* state, long long slot_stride, int state_size,
                                  const int* q_start, const int* state_slots, int n_slots,
                                  float* o_raw, void* scratch, int T, int B, int H, int dk, int dv,
                                  float q_scale, int C, int n_min, int* err,
                                  cudaStream_t stream) {
  CsIn p = {0, (long long)H * dk, 2LL * H * dk, stride, stride, H, H, dk, dv, C, T, B, n_min,
            q_scale};
  if (!cs_sizes_ok(p, state, slot_stride) || state_size % 4 || !gates || !scratch ||
      ((uintptr_t)proj & 7))
    return (int)cudaErrorInvalidValue;
  const __nv_bfloat16* x = (const __nv_bfloat16*)proj;
  return cs_launch<__nv_bfloat16, __nv_bfloat16, true>(
      x, x, p, nullptr, nullptr, gates, state, slot_stride, state_size, q_start, state_slots,
      n_slots, o_raw, (char*)scratch, err, stream);
}
