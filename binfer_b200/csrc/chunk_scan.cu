// Recurrences over a matrix state in chunks of tokens, for the bfloat16 engine's prompt portions:
// what retention.cu (linear scan) and mlstm.cu (matrix memory) walk token by token, as products.
//
//   linear:  S_t = d_t S_{t-1} + k_t v_t^T                        o_t = S_t^T q_t
//   mLSTM:   the same with d_t = exp(f_t + m_{t-1} - m_t), k_t v_t^T times exp(i_t - m_t), a vector
//            n_t beside S_t that takes k_t alone, and o_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6)
//
// With F_t the sum of the log decays up to token t, H_s = F_s - i_s and G_t = min(-m_0, min_{s <= t}
// H_s) (linear: i = m = 0 and G = H = F), token s reaches token t with the weight exp(G_t - H_s)
// (at most 1 unless a decay is above it) and the state before a chunk whose last earlier token is c with
// exp(G_t - G_c); for the mLSTM m_t = F_t - G_t.  F, G and H are double, so a difference of two of them is good to a
// float's last bit; its exponential is a float and what is left of it (cs_exp), the products of q and k
// (and of k and k) inside a chunk are summed in double and rounded once, every other product is float
// (FP32 multiply-adds; on the tensor cores where those files take the sizes: exact products of bfloat16 terms, added
// in float), every sum of one order.  Per chunk of `C` tokens and head:
//
//   cs_gates   F, G, H of every token, its weight behind its chunk; one block per (head, request)
//   cs_qk      Q K^T of a chunk, once per q/k head (several heads may share them), in double
//   cs_state   U = sum_s exp(G_last - H_s) k_s v_s^T: what the chunk adds to the state
//   cs_prefix  from chunk to chunk: S <- exp(G_last - G_c) S + U; U's place takes the state before
//              the chunk; the request's slot takes the last one
//   cs_out     o = [exp(G_t - G_c) q_t | exp(G_t - H_s) (q_t . k_s)] [S ; V]: one product with dk +
//              C terms, the weights applied as its operands are stored into shared memory
//
// The mLSTM with keys in whole steps of 64 and values in whole tiles of 128 runs its products on the tensor
// cores (mlstm_tensor.cuh: the last three kernels become two), and so do the linear scan with keys in whole steps of
// 128, values of 64 or whole tiles of 128 and CTAs enough, and the delta rule with keys of 128 (chunk_tensor.cuh).
//
// GPU time at 2,048 tokens, chunks / walk: 64 heads of 128 x 64 over 8 q/k heads by multiply-adds 208 / 467 us (cs_out
// 99, cs_state 62, cs_prefix 25, cs_qk 14, cs_gates 8), on the tensor cores 133; 8 heads of 128 x 256 117 / 288 (87);
// mLSTM, 8 heads of 256 x 512, 392 / 979 (171, 123, 55, 32, 11; on the tensor cores 212).  What bounds them:
// cs_state and cs_out shared-memory reads (the pipe is 0.61 to 0.64 busy, the multiply-adds 0.3), cs_qk the double
// tensor pipe, cs_prefix memory.  With expf, float products of q and k and the states' sums in runs of 16 these were
// 204, 119 and 381 us, and further from 64 bits than the walk where decays are fast.
//
// Relative errors against 64 bits over 777 tokens, walk / chunks by multiply-adds (chunk_tensor.cuh has those of the
// tensor cores): decays of 0.98 to 1: o 1.9e-7 / 1.4e-7, state 1.8e-7 / 1.3e-7; spread over 0 to 1: o 8.3e-8 /
// 5.0e-8, state 4.0e-8 / 4.2e-8 (half a unit in the last place is up to 6.0e-8); mLSTM, gates that forget in a few
// tokens and in twenty: o 4.8e-7 / 2.3e-7 and 1.3e-5 / 1.2e-6, state 2.9e-8 / 3.7e-8 and 2.3e-7 / 1.0e-7.
//
// Why: the walk has heads x dk x dv independent elements and a chain of multiply-adds from token to
// token, so it left the FP32 pipes at 15 to 20 % (see those files); the products have no chain and
// reach what the float32 product of sgemm_f32.cu reaches.  They are built like it: 64 x 64 outputs
// a CTA, 16 terms a step fetched a step ahead, packed multiply-adds of row pairs.
//
// The gated delta rule, S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q, is the same with u in
// v's place, and the u of a chunk hang together: with F counted from the chunk's start and S0 the state
// before it,  (I + L) U = beta (V - e^F K S0),  L_ts = beta_t exp(F_t - F_s) (k_t . k_s) below the
// diagonal.  So with T = (I + L)^-1:
//
//   cs_qk      K K^T as well
//   ds_prep    per chunk and head: L, T (by blocks of 16), W = T (beta e^F K) and Y = T (beta V)
//   ds_walk    from chunk to chunk: U = Y - W S, S <- exp(F_C) S + K^T (exp(F_C - F) U); leaves U and
//              the states between chunks.  The only chain: two products a chunk, over (request, head,
//              32 columns) in parallel
//   cs_out     as above, on U
//
// 2,048 tokens of 16 heads of 128: 320 us by multiply-adds, 225 on the tensor cores against the walk's 565; 1,000
// tokens 169, 117 and 279, three portions of 1,000 387, 286 and 432.  Errors against 64 bits, walk / multiply-adds:
// keys at random, decays of 0.98 to 1: o 2.3e-7 / 1.6e-7, state 2.3e-7 / 1.8e-7; keys of a cosine of 0.9
// 2.6e-7 / 2.6e-7 and 2.5e-7 / 2.5e-7; fast decays o 1.1e-7 / 7.8e-8, state 6.2e-8 / 7.1e-8.  (What the walk
// has and a chunk's inverse has not is that a token's u answers to the rounding of the one before it:
// where queries, too, lie along what all keys share, a cosine of 0.9 on both sides and slow decays, the
// outputs are 3e-7 from 64 bits and the walk's 0.8e-7.)
//
// Requests of at most `n_min` tokens have no chunks here (the walk serves them).  The order of sums
// depends on where a step's portions begin, so the float32 engine, whose results must not depend
// on the cut, does not use these kernels.
#include "common.cuh"
#include "split_utils.cuh"

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

// v (hi + lo), rounded once
__device__ __forceinline__ float cs_times(float v, float2 w) { return fmaf(v, w.x, v * w.y); }
__device__ __forceinline__ float4 cs_times(float4 v, float2 w) {
  return make_float4(cs_times(v.x, w), cs_times(v.y, w), cs_times(v.z, w), cs_times(v.w, w));
}

// e^x as a float and what is left of it, good to some 2^-26: x = n ln 2 + r in double (n by adding what
// leaves no place for a fraction), the power series of e^r to the seventh power (|r| <= ln 2 / 2: the
// eighth is below 2^-27) on top of 1 + r, whose rounding is kept.  One conversion: those and the double
// operations are what it costs.  (The weights of tokens hang together in every result: with expf, up to two units
// off in the last place, an output of keys and queries alike was four times as far from 64 bits as
// the walk's.)  FINE: with what r's float leaves of it and the eighth power, good to some 2^-27 (2^-29.6 and not
// 2^-27.4 in the mean), for factors: a product of two is then no further off than one exponential.
template <bool FINE = false>
__device__ __forceinline__ float2 cs_exp(double x) {
  if (!(x > -104.0)) return make_float2(x != x ? NAN : 0.f, 0.f);
  if (x > 89.0) return make_float2(INFINITY, 0.f);
  const double whole = 6755399441055744.0;            // 1.5 2^52
  const double t = fma(x, 1.4426950408889634, whole);
  const int n = __double2loint(t);
  const double r = fma(t - whole, -0.69314718055994531, x);
  const float rh = (float)r;
  float q = fmaf(rh, FINE ? fmaf(rh, 1.f / 40320.f, 1.f / 5040.f) : 1.f / 5040.f, 1.f / 720.f);
  q = fmaf(rh, q, 1.f / 120.f);
  q = fmaf(rh, q, 1.f / 24.f);
  q = fmaf(rh, q, 1.f / 6.f);
  q = fmaf(rh, q, 0.5f);
  const float s = 1.f + rh;
  float below = rh - (s - 1.f);
  if (FINE) {
    const float rl = (float)(r - (double)rh);
    below += fmaf(rl, rh, rl);
  }
  const float rest = fmaf(rh * rh, q, below);
  const float hi = s + rest, lo = rest - (hi - s);
  // (two factors: n may lie below the smallest normal exponent)
  const int n1 = n >> 1;
  const float f1 = __int_as_float((n1 + 127) << 23), f2 = __int_as_float((n - n1 + 127) << 23);
  return make_float2(hi * f1 * f2, lo * f1 * f2);
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
#define CS_GATE_THREADS 512

__device__ __forceinline__ double cs_log_decay(float d) {
  // a decay that underflowed to zero forgets everything: exp(-1e4) is zero in float.  One below zero
  // has no logarithm: NaN, like NaN itself (callers leave such decays to the walk)
  return d > 0.f ? fmax(log((double)d), -1e4) : d == 0.f ? -1e4 : (double)NAN;
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
    int n_slots, double* G, double* Hs, float* __restrict__ E,
    double* __restrict__ g0, float2* __restrict__ Wl, int C, int T, int H, int dkdv, int dk, int n_min,
    int decay_stride) {
  __shared__ double sh[CS_GATE_THREADS / 32];
  bf_pdl_trigger();                              // (cs_qk reads nothing of these: it runs beside them)
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
    if (MLSTM) {
      // (-inf, a gate that is shut: exp(-1e5) is zero, and the sums behind it stay numbers)
      const double f = (double)gates[(size_t)(t0 + t) * 2 * H + H + h];
      return f < -1e5 ? -1e5 : f;
    }
    return tok_decay ? cs_log_decay(tok_decay[(size_t)(t0 + t) * decay_stride + h]) : fixed;
  };
  // Wl [H][T]: a token's weight in the state behind its chunk, as a float and what
  // is left, so that a weighted value is rounded once.  (Where decays are fast the state is
  // made up of the last few tokens and the walk rounds little: its state is 4.0e-8 from 64 bits, the
  // chunks' was 4.6e-8 with expf and is 4.2e-8.)
  auto chunk_weights = [&]() {
    __syncthreads();                               // all of g and hs are there
    float2* wl = Wl + (size_t)h * T + t0;
    for (int t = threadIdx.x; t < n; t += CS_GATE_THREADS)
      wl[t] = cs_exp(g[min(n, (t / C + 1) * C) - 1] - hs[t]);
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
    chunk_weights();
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
  chunk_weights();
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

// The same for a step of sixteen tokens whose first is the first of this warp's sixteen rows: row r
// takes the tokens up to its own.  The others' weights are zero, but what they would multiply may be
// an infinity, and a token's result must not depend on the ones behind it.
__device__ __forceinline__ void cs_mul_lower(const float (&As)[CS_K][CS_P],
                                             const float (&Bs)[CS_K][CS_P], int tx, int ty,
                                             CsAcc& total) {
  const int row = (ty & 1) * 8;
  // (a pair of rows at a time: one step of a CTA's, and registers are scarce)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 4
    for (int kk = 0; kk < CS_K; ++kk) {
      const unsigned long long a =
          *reinterpret_cast<const unsigned long long*>(&As[kk][ty * 8 + 2 * i]);
      const float4 w = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
      const unsigned long long b[4] = {cs_pair(w.x, w.x), cs_pair(w.y, w.y), cs_pair(w.z, w.z),
                                       cs_pair(w.w, w.w)};
      const bool both = kk <= row + 2 * i, second = kk == row + 2 * i + 1;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned long long z = cs_fma2(a, b[j], acc[j]);
        if (both) acc[j] = z;
        if (second) acc[j] = (acc[j] & 0xffffffffull) | (z & ~0xffffffffull);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) total[i][j] = cs_add2(total[i][j], acc[j]);
  }
}

// One chain of multiply-adds from step to step, for the states: their sums are rounded as often as the
// walk's there, and a chunk's 64 terms are few.
__device__ __forceinline__ void cs_mul_chain(const float (&As)[CS_K][CS_P],
                                             const float (&Bs)[CS_K][CS_P], int tx, int ty,
                                             CsAcc& acc) {
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
// grid (chunks, QH, row tiles x column tiles): qkm[chunk][qh][C][C] = q_scale Q K^T up to the diagonal
// of every block of 16, and (KK, chunks of one tile) kkm = K K^T.  In double, on the tensor cores
// (mma.sync m8n8k4): a weight inside the chunk is one of these numbers times an exponential, and the
// sums of up to 64 of them behind it show an error that is one of |q| |k|, however small q . k is
// itself.  In float, in runs of 16, outputs were 1.2 to 1.7 times as far from 64 bits as the walk's (fast
// decays; the delta rule's keys alike), at 12 us instead of 14 (2,048 tokens, 8 q/k heads of 128) and 21
// instead of 42 (16 heads, K K^T too, which ds_prep then computed itself in another 5).  A warp takes 16
// rows; of Q alone two warps share a block of 16 rows, every other eight columns each (2,048 tokens of 8 heads of
// 256 33 us with one warp a block, 28 so); the second four warps' blocks run the other way, so that every scheduler
// has the same share of the triangle.
#define CS_QS 32            // sizes a stage
#define CS_QP (CS_QS + 4)   // pitch: eight rows of four neighbouring sizes on different banks

__device__ __forceinline__ void cs_dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// q and k in three bfloat16 terms on the way, for the products on the tensor cores (chunk_tensor.cuh; chunks of 64,
// sizes in whole steps of 64): X[chunk][qh][dk / 64] tiles of three terms of 64 tokens x 64 sizes, a token's sizes
// in a row of 128 bytes with the 128-byte swizzle, rows beyond the chunk's tokens zero.  Numbers without terms
// (split_utils.cuh) are zero; odd[chunk][qh][q | k]: a bit for every token that has one.
struct CsTerms {
  uint8_t *q, *k;              // (null: not asked for)
  unsigned long long* odd;
};
#define CS_TERMS_TERM (64 * 128)
#define CS_TERMS_TILE (3 * CS_TERMS_TERM)
// the first float that has none, times 2^24, as bits
constexpr uint32_t CS_NO_TERMS_UP = 0x7f7f8000u - (24u << 23);
// four sizes of a token; true where one has no terms
__device__ __forceinline__ bool cs_put_terms(uint8_t* X, int token, int size, float4 v) {
  float x[4] = {v.x, v.y, v.z, v.w};
  bool bad = false;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if ((__float_as_uint(x[i]) & 0x7fffffffu) >= CS_NO_TERMS_UP) {
      bad = true;
      x[i] = 0.f;
    }
  uint2 hi, mid, lo;
  split_up(x[0], x[1]);
  split_up(x[2], x[3]);
  split3(x[0], x[1], hi.x, mid.x, lo.x);
  split3(x[2], x[3], hi.y, mid.y, lo.y);
  uint8_t* to = X + (size_t)(size >> 6) * CS_TERMS_TILE + token * 128 + ((((size >> 3) & 7) ^ (token & 7)) << 4) +
                (size & 4) * 2;
  *reinterpret_cast<uint2*>(to) = hi;
  *reinterpret_cast<uint2*>(to + CS_TERMS_TERM) = mid;
  *reinterpret_cast<uint2*>(to + 2 * CS_TERMS_TERM) = lo;
  return bad;
}
// Two blocks beside those of a chunk and head's products, which the double tensor pipe bounds, where these are
// bound by memory: q's terms (what 0) and k's.
template <int THREADS>
__device__ __forceinline__ void cs_terms(const float* __restrict__ qk, const CsIn& p, const CsChunk& c, int what,
                                         const CsTerms& out) {
  __shared__ unsigned long long odd;
  if (threadIdx.x == 0) odd = 0ull;
  __syncthreads();
  const int at = c.index * 64, n = min(64, c.n - at), pieces = p.dk / 8;
  const float* rows = qk + (size_t)(c.t0 + at) * p.qk_stride + (what ? p.k_off : p.q_off) + (size_t)blockIdx.y * p.dk;
  const size_t head = (size_t)blockIdx.x * p.QH + blockIdx.y;
  uint8_t* X = (what ? out.k : out.q) + head * (p.dk / 64) * CS_TERMS_TILE;
#pragma unroll 4
  for (int i = threadIdx.x; i < 64 * pieces; i += THREADS) {
    const int t = i / pieces, pc = i % pieces;
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (t < n) {
      const float4 a = *reinterpret_cast<const float4*>(rows + (size_t)t * p.qk_stride + 8 * pc);
      const float4 b = *reinterpret_cast<const float4*>(rows + (size_t)t * p.qk_stride + 8 * pc + 4);
      x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
    }
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if ((__float_as_uint(x[j]) & 0x7fffffffu) >= CS_NO_TERMS_UP) {
        bad = true;
        x[j] = 0.f;
      }
    if (bad) atomicOr(&odd, 1ull << t);
    uint4 hi, mid, lo;
#pragma unroll
    for (int j = 0; j < 8; j += 2) split_up(x[j], x[j + 1]);
    split3(x[0], x[1], hi.x, mid.x, lo.x);
    split3(x[2], x[3], hi.y, mid.y, lo.y);
    split3(x[4], x[5], hi.z, mid.z, lo.z);
    split3(x[6], x[7], hi.w, mid.w, lo.w);
    uint8_t* to = X + (size_t)(pc >> 3) * CS_TERMS_TILE + t * 128 + (((pc & 7) ^ (t & 7)) << 4);
    *reinterpret_cast<uint4*>(to) = hi;
    *reinterpret_cast<uint4*>(to + CS_TERMS_TERM) = mid;
    *reinterpret_cast<uint4*>(to + 2 * CS_TERMS_TERM) = lo;
  }
  __syncthreads();
  if (threadIdx.x == 0) out.odd[head * 2 + what] = odd;
}

template <typename A, bool KK>
__global__ void __launch_bounds__(256) cs_qk_kernel(
    const A* __restrict__ qk, CsIn p, const int* __restrict__ q_start, float* __restrict__ qkm,
    float* __restrict__ kkm, CsTerms x_out) {
  constexpr int THREADS = 256, PIECES = 128 * (CS_QS / 4) / THREADS, SHARES = KK ? 1 : 2, COLS = 8 / SHARES;
  __shared__ __align__(16) double rows_s[128][CS_QP];      // 64 rows of q, 64 of k
  const int tiles = p.C / CS_T;
  const int rt = blockIdx.z / tiles, ct = blockIdx.z % tiles;
  const CsChunk c = cs_find(q_start, p.B, p.C, p.n_min, blockIdx.x, -1);
  const int at = c.index * p.C;                  // the chunk's first token inside the request
  const int n = min(p.C, c.n - at);
  if constexpr (sizeof(A) == 4) {
    if (rt >= tiles && c.b >= 0) cs_terms<THREADS>(qk, p, c, blockIdx.z - tiles * tiles, x_out);
  }
  if (ct > rt || c.b < 0 || rt * CS_T >= n || rt >= tiles) {
    bf_pdl_wait();                               // (on every path: this grid's end is that of cs_gates, too)
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hq = blockIdx.y;
  const A* q = qk + (size_t)(c.t0 + at) * p.qk_stride + p.q_off + (size_t)hq * p.dk;
  const A* k = qk + (size_t)(c.t0 + at) * p.qk_stride + p.k_off + (size_t)hq * p.dk;
  const bool of_k = KK && warp >= 4;             // rows of K against K
  const int share = KK ? 0 : warp >> 2, block = warp >= 4 ? 7 - warp : warp;
  const int row0 = (of_k ? 64 : 0) + block * 16;
  const int cols = ct < rt ? 8 : 2 * (block + 1);          // blocks of eight columns: this warp's shares of them
  double acc[2][COLS][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  float4 f[PIECES];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int x = 0; x < PIECES; ++x) {
      const int idx = tid + x * THREADS, r = idx / (CS_QS / 4), kk = k0 + idx % (CS_QS / 4) * 4;
      const int row = (r < 64 ? rt : ct) * CS_T + (r & 63);
      f[x] = row < n && kk < p.dk ? cs_ld4((r < 64 ? q : k) + (size_t)row * p.qk_stride + kk)
                                  : cs_zero();
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < p.dk; k0 += CS_QS) {
#pragma unroll
    for (int x = 0; x < PIECES; ++x) {
      const int idx = tid + x * THREADS;
      double2* d = reinterpret_cast<double2*>(&rows_s[idx / (CS_QS / 4)][idx % (CS_QS / 4) * 4]);
      d[0] = make_double2(f[x].x, f[x].y);
      d[1] = make_double2(f[x].z, f[x].w);
    }
    __syncthreads();
    if (k0 + CS_QS < p.dk) fetch(k0 + CS_QS);
#pragma unroll 2
    for (int kk = 0; kk < CS_QS; kk += 4) {
      const double a0 = rows_s[row0 + (lane >> 2)][kk + (lane & 3)];
      const double a1 = rows_s[row0 + 8 + (lane >> 2)][kk + (lane & 3)];
#pragma unroll
      for (int j = 0; j < COLS; ++j)
        if (SHARES * j + share < cols) {
          const double b = rows_s[64 + 8 * (SHARES * j + share) + (lane >> 2)][kk + (lane & 3)];
          cs_dmma(acc[0][j], a0, b);
          cs_dmma(acc[1][j], a1, b);
        }
    }
    __syncthreads();
  }
  const double scale = of_k ? 1.0 : (double)p.q_scale;
  float* dst = (of_k ? kkm : qkm) + ((size_t)blockIdx.x * p.QH + hq) * p.C * p.C;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < COLS; ++j)
      if (SHARES * j + share < cols)
        *reinterpret_cast<float2*>(
            dst + (size_t)(rt * CS_T + block * 16 + 8 * i + (lane >> 2)) * p.C + ct * CS_T + 8 * (SHARES * j + share) +
            (lane & 3) * 2) = make_float2((float)(acc[i][j][0] * scale), (float)(acc[i][j][1] * scale));
  bf_pdl_wait();
}

// ------------------------------------------------------------------------------- cs_state
// grid (chunks, H, row tiles x column tiles).  U[chunk][h]: linear [dv][dk], mLSTM [dk][dv] (each
// like its state); mLSTM: Un[chunk][h][dk] by the CTAs of the first column tile.
template <typename A, typename V, bool MLSTM>
__global__ void __launch_bounds__(CS_THREADS, 4) cs_state_kernel(
    const A* __restrict__ qk, const V* __restrict__ vsrc, CsIn p, const int* __restrict__ q_start,
    const float2* __restrict__ Wl, float* __restrict__ U, float* __restrict__ Un) {
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
  const float2* wl = Wl + (size_t)h * p.T + c.t0 + at;
  CsAcc acc;
  cs_clear(acc);
  float nacc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) nacc[i] = 0.f;
  float4 fk[2], fv[2];
  float2 fw[2];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int idx = tid + x * CS_THREADS, s = s0 + (idx >> 4), d = (idx & 15) * 4;
      const int dkk = (MLSTM ? r0 : c0) + d, dvv = (MLSTM ? c0 : r0) + d;
      fw[x] = s < n ? wl[s] : make_float2(0.f, 0.f);
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
      if (MLSTM && (idx & 15) == 0) ws[buf][idx >> 4] = fw[x].x;
    }
  };
  fetch(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int s0 = 0; s0 < n; s0 += CS_K, buf ^= 1) {
    if (s0 + CS_K < n) fetch(s0 + CS_K);
    cs_mul_chain(As[buf], Bs[buf], tx, ty, acc);
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
        const float2 d = cs_exp(last - before);
        before = last;
        S = make_float4(fmaf(d.x, S.x, fmaf(d.y, S.x, add.x)), fmaf(d.x, S.y, fmaf(d.y, S.y, add.y)),
                        fmaf(d.x, S.z, fmaf(d.y, S.z, add.z)), fmaf(d.x, S.w, fmaf(d.y, S.w, add.w)));
      }
    }
  }
  *reinterpret_cast<float4*>(s_at) = S;
}

// ---------------------------------------------------------------------------------- cs_out
// grid (chunks, H, row tiles x column tiles of dv)
// KROWS: a chunk's state lies as [dk][dv] (the mLSTM's, and what ds_walk leaves), else [dv][dk]
template <typename A, typename V, bool MLSTM, bool KROWS>
__global__ void __launch_bounds__(CS_THREADS, 4) cs_out_kernel(
    const A* __restrict__ qk, const V* __restrict__ vsrc, CsIn p, const int* __restrict__ q_start,
    const int* __restrict__ state_slots, int n_slots, const double* __restrict__ G,
    const double* __restrict__ Hs, const double* __restrict__ g0, const float* __restrict__ E,
    const float* __restrict__ qkm, const float* __restrict__ U, const float* __restrict__ Un,
    float* __restrict__ o_raw) {
  __shared__ __align__(16) float As[2][CS_K][CS_P], Bs[2][CS_K][CS_P];
  __shared__ double gt[CS_T];
  __shared__ float2 at_s[CS_T];
  __shared__ float ns[2][CS_K];
  __shared__ int odd[2];        // the step whose values in this buffer are not all finite
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
    float2 w = make_float2(0.f, 0.f);
    if (r0 + tid < n) {
      w = cs_exp(x - before);
      // (times q_scale: its products' roundings are part of what is left)
      const float f = w.x * p.q_scale;
      w = make_float2(f, fmaf(w.x, p.q_scale, -f) + w.y * p.q_scale);
      if (!(fabsf(f) < INFINITY)) w.y = 0.f;
    }
    at_s[tid] = w;
  }
  if (tid < 2) odd[tid] = -1;
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
        if (KROWS) {                           // S [dk][dv]: rows of terms
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
        if (KROWS) cs_put(Bs[buf], idx, fb[x]);
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
        float4 w = cs_zero();
        if (s <= last) {
          w.x = cs_times(fa[x].x, cs_exp(gr - fh[0]));
          if (s + 1 <= last) w.y = cs_times(fa[x].y, cs_exp(gr - fh[1]));
          if (s + 2 <= last) w.z = cs_times(fa[x].z, cs_exp(gr - fh[2]));
          if (s + 3 <= last) w.w = cs_times(fa[x].w, cs_exp(gr - fh[3]));
        }
        // (a number times zero is zero if it is finite, and only then)
        if (!(fb[x].x * 0.f + fb[x].y * 0.f + fb[x].z * 0.f + fb[x].w * 0.f == 0.f)) odd[buf] = k0;
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
    // the tokens before, among and behind this warp's sixteen rows
    const int ahead = k0 < dk_pad ? -1 : k0 - dk_pad - ((ty & ~1) * 8 + r0);
    if (ahead < 0) cs_mul(As[buf], Bs[buf], tx, ty, acc);
    else if (ahead == 0 && odd[buf] != k0) cs_mul(As[buf], Bs[buf], tx, ty, acc);
    else if (ahead == 0) cs_mul_lower(As[buf], Bs[buf], tx, ty, acc);
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

#include "mlstm_tensor.cuh"

struct DsIn {
  const float* qkv;        // [T][C]: q (G heads of dk), k, v (H heads of dv)
  const float* gates;      // [T][2][H]: beta, decay
  long long stride;        // C
  int H, G, dk, dv, T, B, n_min;
};

__device__ __forceinline__ void ds_cp16(float* smem, const float* gmem, bool ok) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(gmem),
               "r"(ok ? 16 : 0));
}

#include "chunk_tensor.cuh"

// ------------------------------------------------------------------- the gated delta rule
#define DS_C 64            // tokens a chunk
#define DS_D 128           // most key and value sizes
#define DS_P (DS_D + 4)
#define DS_NS 32           // columns of the state a CTA of ds_walk keeps
#define DS_PREP_THREADS 256

// four of L's numbers, all left of the diagonal, with exponentials of their own
__device__ __noinline__ void ds_again_L(const double* fs, float beta, int t, int s, float4 kk, float* out) {
  const float xs[4] = {kk.x, kk.y, kk.z, kk.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 w = cs_exp(fs[t] - fs[s + j]);
    out[j] = (float)((double)beta * ((double)w.x + (double)w.y) * (double)xs[j]);
  }
}

// grid (chunks, H): W [chunk][H][64][dk], Y [chunk][H][64][dv]
// 1,111 and 694 tokens of 16 heads of 128: 39 us, 54 before (without terms and weights, 16 heads of
// 64: 35, 46).  A block's phases follow one another (26,000 cycles, two blocks an SM), so it is the length of each that
// counts: L's exponentials as products of the factors that the outputs' weights have anyway 7,400 -> 2,200 cycles; T's
// rows with a thread at one row and column of each block, loops unrolled, 9,700 -> 3,100; the decays asked for ahead of
// keys and values 3 us; W and Y with even shares for the schedulers 4,900 -> 4,100.
__global__ void __launch_bounds__(DS_PREP_THREADS, 2) ds_prep_kernel(
    DsIn p, const int* __restrict__ q_start, const double* __restrict__ F,
    const float* __restrict__ KKm, float* __restrict__ W, float* __restrict__ Y,
    const float* __restrict__ qkm, CtHead* __restrict__ Ww, uint8_t* __restrict__ Xw,
    unsigned long long* __restrict__ odd_w) {
  extern __shared__ __align__(16) float ds_smem[];
  __shared__ unsigned long long odd;
  float* Ks = ds_smem;                           // [64][DS_P]
  float* Vs = Ks + DS_C * DS_P;                  // [64][DS_P]
  float* Ls = Vs + DS_C * DS_P;                  // [64][68]
  float* Ts = Ls + DS_C * 68;                    // [64][68]
  float* Rs = Ts + DS_C * 68;                    // [16][52]
  __shared__ double fs[DS_C];
  __shared__ float beta[DS_C], grow[DS_C];       // grow: beta e^F
  const CsChunk c = cs_find(q_start, p.B, DS_C, p.n_min, blockIdx.x, -1);
  if (c.b < 0) return;
  const int at = c.index * DS_C, n = min(DS_C, c.n - at);
  const int h = blockIdx.y, hq = h / (p.H / p.G);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const float* k = p.qkv + (size_t)(c.t0 + at) * p.stride + (size_t)(p.G + hq) * p.dk;
  const float* v = p.qkv + (size_t)(c.t0 + at) * p.stride + 2 * (size_t)p.G * p.dk + (size_t)h * p.dv;
  // (the few numbers that are waited for first are asked for first)
  const double* f = F + (size_t)h * p.T + c.t0 + at;
  const double f0 = c.index ? f[-1] : 0.0, f_t = tid < n ? f[tid] : 0.0;
  const float beta_t = tid < n ? p.gates[(size_t)(c.t0 + at + tid) * 2 * p.H + h] : 0.f;
  for (int i = tid; i < DS_C * (DS_D / 4); i += DS_PREP_THREADS) {
    const int r = i / (DS_D / 4), e = i % (DS_D / 4) * 4;
    const bool ok_k = r < n && e < p.dk, ok_v = r < n && e < p.dv;
    ds_cp16(Ks + r * DS_P + e, ok_k ? k + (size_t)r * p.stride + e : p.qkv, ok_k);
    ds_cp16(Vs + r * DS_P + e, ok_v ? v + (size_t)r * p.stride + e : p.qkv, ok_v);
  }
  asm volatile("cp.async.commit_group;" ::);
  if (tid < DS_C) {
    fs[tid] = f_t;
    beta[tid] = beta_t;
    grow[tid] = cs_times(beta_t, cs_exp(tid < n ? f_t - f0 : 0.0));
  }
  if (tid == 0) odd = 0ull;
  __syncthreads();
  // exp(F_t - F_s) for L, and for the outputs' weights; the tables lie where T will
  static_assert(sizeof(CtWeights) <= DS_C * 68 * sizeof(float), "");
  CtWeights& tab = *reinterpret_cast<CtWeights*>(Ts);
  CtHead* head = Ww ? Ww + (size_t)blockIdx.x * p.H + h : nullptr;
  const bool above = ct_factors(fs, fs, f0, n, 1.f, tab, head ? head->at : nullptr);
  if (head) ct_weights(tab, n, above, qkm + ((size_t)blockIdx.x * p.G + hq) * DS_C * DS_C, head);
  const float* kk = KKm + ((size_t)blockIdx.x * p.G + hq) * DS_C * DS_C;
  float4 kt[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) kt[i] = *reinterpret_cast<const float4*>(kk + (ty * 4 + i) * DS_C + 4 * tx);
  asm volatile("cp.async.wait_group 0;" ::);
  __syncthreads();
  // L: rows 4 ty .., columns 4 tx .., rounded once (keys alike make it hang on every bit)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty * 4 + i;
    const float4 x = kt[i];
    const int bl = tx >> 2;                      // the block of 16 that s is in
    const bool own = bl == t >> 4, some = 4 * tx < t && t < n;
    const float4 hi = *reinterpret_cast<const float4*>(own ? &tab.near[0][t][4 * tx & 15] : &tab.col[0][4 * tx % 48]);
    const float4 lo = *reinterpret_cast<const float4*>(own ? &tab.near[1][t][4 * tx & 15] : &tab.col[1][4 * tx % 48]);
    const double by = (double)beta[t] * (own || !some ? 1.0 : (double)tab.row[0][bl][t] + (double)tab.row[1][bl][t]);
    auto one = [&](float k2, float whi, float wlo, int j) {
      return some && 4 * tx + j < t ? (float)(by * ((double)whi + (double)wlo) * (double)k2) : 0.f;
    };
    if (above && !own && some) {
      ds_again_L(fs, beta[t], t, 4 * tx, x, Ls + t * 68 + 4 * tx);
      continue;
    }
    *reinterpret_cast<float4*>(Ls + t * 68 + 4 * tx) =
        make_float4(one(x.x, hi.x, lo.x, 0), one(x.y, hi.y, lo.y, 1), one(x.z, hi.z, lo.z, 2),
                    one(x.w, hi.w, lo.w, 3));
  }
  __syncthreads();
  // T = (I + L)^-1 by blocks of 16: the diagonal blocks, a thread a column ...
  for (int i = tid; i < DS_C * 68; i += DS_PREP_THREADS) Ts[i] = 0.f;
  __syncthreads();
  if (tid < DS_C) {
    const int o = tid & ~15, j = tid & 15;
    float col[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      float r = t == j ? 1.f : 0.f;
#pragma unroll
      for (int s = 0; s < t; s += 4) {
        const float4 l = *reinterpret_cast<const float4*>(Ls + (o + t) * 68 + o + s);
        r = fmaf(-l.x, col[s], r);
        if (s + 1 < t) r = fmaf(-l.y, col[s + 1], r);
        if (s + 2 < t) r = fmaf(-l.z, col[s + 2], r);
        if (s + 3 < t) r = fmaf(-l.w, col[s + 3], r);
      }
      col[t] = r;
      Ts[(o + t) * 68 + o + j] = r;
    }
  }
  __syncthreads();
  // ... then block row by block row: T_i* = -T_ii (sum_k L_ik T_k*), a thread row ty, column tx of each block
#pragma unroll
  for (int i = 1; i < 4; ++i) {
    const float* l = Ls + (16 * i + ty) * 68;
    float a0[3] = {0.f, 0.f, 0.f}, a1[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 16 * i; s += 4) {
      const float4 x = *reinterpret_cast<const float4*>(l + s);
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (16 * b > s) continue;                // (T is zero there, but x may be infinite)
        const float* t = Ts + s * 68 + 16 * b + tx;
        a0[b] = fmaf(x.x, t[0], a0[b]);
        a1[b] = fmaf(x.y, t[68], a1[b]);
        a0[b] = fmaf(x.z, t[2 * 68], a0[b]);
        a1[b] = fmaf(x.w, t[3 * 68], a1[b]);
      }
    }
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (b < i) Rs[ty * 52 + 16 * b + tx] = a0[b] + a1[b];
    __syncthreads();
    float a[3] = {0.f, 0.f, 0.f};
    float* t = Ts + (16 * i + ty) * 68;
#pragma unroll
    for (int s4 = 0; s4 < 16; s4 += 4) {
      const float4 x = *reinterpret_cast<const float4*>(t + 16 * i + s4);
      const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // (row s of the block reaches the rows from s on alone, also where it is not finite)
        if (s4 + j > ty) continue;
#pragma unroll
        for (int b = 0; b < 3; ++b)
          if (b < i) a[b] = fmaf(xs[j], Rs[(s4 + j) * 52 + 16 * b + tx], a[b]);
      }
    }
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (b < i) t[16 * b + tx] = -a[b];
    __syncthreads();
  }
  // W = T (beta e^F K), Y = T (beta V): rows 4 r4 .., columns 4 tx + 64 j.  (Row block r4 has r4 + 1 of 16 terms:
  // warps w and w + 4, of one scheduler, have 34 between them whatever w is)
  const int r4 = ty < 8 ? ty : 23 - ty;
#pragma unroll 1
  for (int what = 0; what < 2; ++what) {
    const float* B = what ? Vs : Ks;
    const float* sc = what ? beta : grow;
    const int width = what ? p.dv : p.dk;
    unsigned long long acc[4][2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0ull;
    // (T is zero above the diagonal, but what stands there may be infinite: a thread's last four terms
    // are those that its rows have)
    auto four = [&](int s, bool last) {
      float4 tr[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        tr[i] = *reinterpret_cast<const float4*>(Ts + (r4 * 4 + i) * 68 + s);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float fsc = sc[s + x];
        ulonglong2 b[2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
          b[j] = *reinterpret_cast<const ulonglong2*>(B + (s + x) * DS_P + 4 * tx + 64 * j);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (last && i < x) continue;
          const float w = (x == 0 ? tr[i].x : x == 1 ? tr[i].y : x == 2 ? tr[i].z : tr[i].w) * fsc;
          const unsigned long long w2 = cs_pair(w, w);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            acc[i][j][0] = cs_fma2(w2, b[j].x, acc[i][j][0]);
            acc[i][j][1] = cs_fma2(w2, b[j].y, acc[i][j][1]);
          }
        }
      }
    };
    for (int s = 0; s < r4 * 4; s += 4) four(s, false);
    four(r4 * 4, true);
    float* dst = (what ? Y : W) + ((size_t)blockIdx.x * p.H + h) * DS_C * width;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int col = 4 * tx + 64 * j;
        if (col >= width) continue;
        float4 r;
        cs_unpair(acc[i][j][0], r.x, r.y);
        cs_unpair(acc[i][j][1], r.z, r.w);
        *reinterpret_cast<float4*>(dst + (size_t)(r4 * 4 + i) * width + col) = r;
        // W in terms, too, for dt_walk
        if (Xw && !what && cs_put_terms(Xw + ((size_t)blockIdx.x * p.H + h) * 2 * CS_TERMS_TILE, r4 * 4 + i, col, r))
          atomicOr(&odd, 1ull << (r4 * 4 + i));
      }
  }
  if (Xw) {
    __syncthreads();
    if (tid == 0) odd_w[(size_t)blockIdx.x * p.H + h] = odd;
  }
}

// grid (column slices of 32, H, B): u [T][H][dv], Sc [chunk][H][dk][dv] (the state before each chunk).
// 128 threads with 4 x 4 outputs of U and 8 x 4 of the state each: what a thread reads from shared
// memory (at 128 bytes a cycle and SM) is about what its multiply-adds take.  1,111 and 694 tokens of
// 16 heads of 64: 86 us.  (By 16 heads of 128, which dt_walk takes unless its scratch is too much: 108 us; the
// choices were made there, at 115: 256 threads with half of that 130, and the state's columns in the lanes'
// registers, W and K read by all lanes alike, 133.)
__global__ void __launch_bounds__(128) ds_walk_kernel(
    DsIn p, const int* __restrict__ q_start, const int* __restrict__ state_slots, int n_slots,
    float* __restrict__ state, long long slot_stride, const double* __restrict__ F,
    const float2* __restrict__ Wl, const float* __restrict__ W, const float* __restrict__ Y,
    float* __restrict__ u,
    float* __restrict__ Sc, int* __restrict__ err) {
  extern __shared__ __align__(16) float ds_smem[];
  constexpr int PS = DS_NS + 4;
  float* Ws = ds_smem;                           // [2][64][DS_P]
  float* Ks = Ws + 2 * DS_C * DS_P;              // [2][64][DS_P]
  float* Ss = Ks + 2 * DS_C * DS_P;              // [DS_D][PS]
  float* Us = Ss + DS_D * PS;                    // [64][PS]: exp(F_C - F_s) u_s
  const int h = blockIdx.y, b = blockIdx.z, col0 = blockIdx.x * DS_NS;
  const CsChunk c = cs_find(q_start, p.B, DS_C, p.n_min, 0, b);
  if (c.n <= p.n_min) return;
  const int slot = state_slots[b];
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;   // 8 x 16
  if (slot < 0 || slot >= n_slots) {
    if (tid == 0) atomicOr(err, BF_ERR_SLOT);
    return;
  }
  const int hq = h / (p.H / p.G);
  float* st = state + (size_t)slot * slot_stride + (size_t)h * p.dv * p.dk;
  const float* k = p.qkv + (size_t)c.t0 * p.stride + (size_t)(p.G + hq) * p.dk;
  const double* f = F + (size_t)h * p.T + c.t0;
  const float2* wl = Wl + (size_t)h * p.T + c.t0;
  const int chunks = (c.n + DS_C - 1) / DS_C;
  auto load = [&](int i, int buf) {
    const int n = min(DS_C, c.n - i * DS_C);
    const float* w = W + ((size_t)(c.first + i) * p.H + h) * DS_C * p.dk;
    for (int e = tid; e < DS_C * (DS_D / 4); e += 128) {
      const int r = e / (DS_D / 4), d = e % (DS_D / 4) * 4;
      const bool ok = d < p.dk, ok_k = ok && r < n;
      ds_cp16(Ws + (buf * DS_C + r) * DS_P + d, ok ? w + (size_t)r * p.dk + d : W, ok);
      ds_cp16(Ks + (buf * DS_C + r) * DS_P + d,
              ok_k ? k + (size_t)(i * DS_C + r) * p.stride + d : p.qkv, ok_k);
    }
    asm volatile("cp.async.commit_group;" ::);
  };
  load(0, 0);
  for (int e = tid; e < DS_D * DS_NS; e += 128) {
    const int kk = e % DS_D, j = e / DS_D;
    Ss[kk * PS + j] = kk < p.dk && col0 + j < p.dv ? st[(size_t)(col0 + j) * p.dk + kk] : 0.f;
  }
  // this thread's state: rows 8 ty .. 8 ty + 7 (four pairs), columns 4 tx ..; U: rows 4 ty ..
  const int col = col0 + 4 * tx;
  double before = 0.0;
  for (int i = 0; i < chunks; ++i) {
    const int n = min(DS_C, c.n - i * DS_C);
    const float* Wt = Ws + (i & 1) * DS_C * DS_P;
    const float* Kt = Ks + (i & 1) * DS_C * DS_P;
    const double last = f[i * DS_C + n - 1];
    asm volatile("cp.async.wait_group 0;" ::);
    __syncthreads();                             // the chunk and the state are here
    if (i + 1 < chunks) load(i + 1, (i + 1) & 1);
    const size_t chunk = (size_t)(c.first + i) * p.H + h;
    float4 y[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
      y[r] = col < p.dv ? *reinterpret_cast<const float4*>(
                              Y + (chunk * DS_C + ty * 4 + r) * p.dv + col)
                        : cs_zero();
    // the state before the chunk, for cs_out
    if (col < p.dv) {
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (ty * 8 + r < p.dk)
          *reinterpret_cast<float4*>(Sc + (chunk * p.dk + ty * 8 + r) * p.dv + col) =
              *reinterpret_cast<const float4*>(Ss + (ty * 8 + r) * PS + 4 * tx);
    }
    // U = Y - W S, in runs of 16 terms
    unsigned long long tot[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) tot[r][0] = tot[r][1] = 0ull;
#pragma unroll 1
    for (int d0 = 0; d0 < p.dk; d0 += 16) {
      unsigned long long acc[4][2];
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0ull;
#pragma unroll
      for (int d = d0; d < d0 + 16; d += 4) {
        float4 w[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          w[r] = *reinterpret_cast<const float4*>(Wt + (ty * 4 + r) * DS_P + d);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const ulonglong2 sv = *reinterpret_cast<const ulonglong2*>(Ss + (d + x) * PS + 4 * tx);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float wv = x == 0 ? w[r].x : x == 1 ? w[r].y : x == 2 ? w[r].z : w[r].w;
            const unsigned long long w2 = cs_pair(wv, wv);
            acc[r][0] = cs_fma2(w2, sv.x, acc[r][0]);
            acc[r][1] = cs_fma2(w2, sv.y, acc[r][1]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        tot[r][0] = cs_add2(tot[r][0], acc[r][0]);
        tot[r][1] = cs_add2(tot[r][1], acc[r][1]);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = ty * 4 + r;
      float4 a;
      cs_unpair(tot[r][0], a.x, a.y);
      cs_unpair(tot[r][1], a.z, a.w);
      const float4 uv = make_float4(y[r].x - a.x, y[r].y - a.y, y[r].z - a.z, y[r].w - a.w);
      const float2 g = t < n ? wl[i * DS_C + t] : make_float2(0.f, 0.f);
      *reinterpret_cast<float4*>(Us + t * PS + 4 * tx) = cs_times(uv, g);
      if (t < n && col < p.dv)
        *reinterpret_cast<float4*>(u + ((size_t)(c.t0 + i * DS_C + t) * p.H + h) * p.dv + col) = uv;
    }
    __syncthreads();                             // U is whole; the state before it is read
    // S <- exp(F_C) S + K^T U, one chain (rounded as often as the walk's)
    unsigned long long S[4][4];
    const float2 g = cs_exp(last - before);
    before = last;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        S[r][j] = cs_pair(cs_times(Ss[(ty * 8 + 2 * r) * PS + 4 * tx + j], g),
                          cs_times(Ss[(ty * 8 + 2 * r + 1) * PS + 4 * tx + j], g));
#pragma unroll 1
    for (int s0 = 0; s0 < n; s0 += 16) {         // (rows of Us and Ks from n on are zero)
#pragma unroll
      for (int s = s0; s < s0 + 16; ++s) {
        const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(Kt + s * DS_P + ty * 8);
        const ulonglong2 k1 = *reinterpret_cast<const ulonglong2*>(Kt + s * DS_P + ty * 8 + 4);
        const float4 uv = *reinterpret_cast<const float4*>(Us + s * PS + 4 * tx);
        const unsigned long long a[4] = {k0.x, k0.y, k1.x, k1.y};
        const unsigned long long w[4] = {cs_pair(uv.x, uv.x), cs_pair(uv.y, uv.y),
                                         cs_pair(uv.z, uv.z), cs_pair(uv.w, uv.w)};
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int j = 0; j < 4; ++j) S[r][j] = cs_fma2(a[r], w[j], S[r][j]);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        cs_unpair(S[r][j], Ss[(ty * 8 + 2 * r) * PS + 4 * tx + j],
                  Ss[(ty * 8 + 2 * r + 1) * PS + 4 * tx + j]);
  }
  __syncthreads();
  for (int e = tid; e < DS_D * DS_NS; e += 128) {
    const int kk = e % DS_D, j = e / DS_D;
    if (kk < p.dk && col0 + j < p.dv) st[(size_t)(col0 + j) * p.dk + kk] = Ss[kk * PS + j];
  }
}

// -------------------------------------------------------------------------------- launches
// Scratch (bytes, each part on a 256-byte boundary): G, Hs, g0, Wl | E (mLSTM) | qkm | U | Un
// (mLSTM) | Xq, Xk, odd, W (`terms`: chunk_tensor.cuh).
struct CsLayout {
  size_t G, Hs, g0, Wl, E, qkm, U, Un, Xq, Xk, odd, W, total;
  int chunks;
};
// The most chunks of C tokens that a step's portions of more than n_min tokens can have.
static int cs_most_chunks(int T, int B, int C, int n_min) {
  const int long_ones = T / (n_min + 1);
  return T / C + (B < long_ones ? B : long_ones);
}
static CsLayout cs_layout(int T, int B, int H, int QH, int dk, int dv, int C, int mlstm,
                          int n_min, bool terms) {
  CsLayout l;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 255) & ~(size_t)255;
    return here;
  };
  l.chunks = cs_most_chunks(T, B, C, n_min);
  l.G = take((size_t)T * H * 8);
  l.Hs = take((size_t)T * H * 8);
  l.g0 = take((size_t)B * H * 8);
  l.Wl = take((size_t)T * H * 8);
  l.E = take(mlstm ? (size_t)T * H * 4 : 0);
  l.qkm = take((size_t)l.chunks * QH * C * C * 4);
  l.U = take((size_t)l.chunks * H * dk * dv * 4);
  l.Un = take(mlstm ? (size_t)l.chunks * H * dk * 4 : 0);
  l.Xq = take(terms ? ct_terms_bytes(l.chunks, QH, dk) : 0);
  l.Xk = take(terms ? ct_terms_bytes(l.chunks, QH, dk) : 0);
  l.odd = take(terms ? (size_t)l.chunks * QH * 16 : 0);
  l.W = take(terms ? (size_t)l.chunks * H * sizeof(CtHead) : 0);
  l.total = at;
  return l;
}

// terms: with the room that a linear scan's products on the tensor cores need (0 where none takes the sizes)
BF_EXPORT long long bf_chunk_scan_scratch(int T, int B, int H, int QH, int dk, int dv, int C,
                                          int mlstm, int n_min, int terms) {
  if (terms && (mlstm || !ct_takes(H, QH, dk, dv, C, cs_most_chunks(T, B, C, n_min)))) return 0;
  return (long long)cs_layout(T, B, H, QH, dk, dv, C, mlstm, n_min, terms).total;
}

template <typename A, typename V, bool MLSTM>
static int cs_launch(const A* qk, const V* v, const CsIn& p, const float* decays,
                     const float* tok_decay, const float* gates, float* state,
                     long long slot_stride, int state_size, const int* q_start,
                     const int* state_slots, int n_slots, float* o_raw, char* scratch, int* err,
                     cudaStream_t stream, bool tensor = false) {
  const CsLayout l = cs_layout(p.T, p.B, p.H, p.QH, p.dk, p.dv, p.C, MLSTM, p.n_min, !MLSTM && tensor);
  double* G = (double*)(scratch + l.G);
  double* Hs = (double*)(scratch + l.Hs);
  double* g0 = (double*)(scratch + l.g0);
  float2* Wl = (float2*)(scratch + l.Wl);
  float* E = (float*)(scratch + l.E);
  float* qkm = (float*)(scratch + l.qkm);
  float* U = (float*)(scratch + l.U);
  float* Un = (float*)(scratch + l.Un);
  const int tiles = p.C / CS_T, tk = (p.dk + CS_T - 1) / CS_T, tv = (p.dv + CS_T - 1) / CS_T;
  cs_gates_kernel<MLSTM><<<dim3(p.H, p.B), CS_GATE_THREADS, 0, stream>>>(
      decays, tok_decay, gates, state, slot_stride, state_size, q_start, state_slots, n_slots, G,
      Hs, E, g0, Wl, p.C, p.T, p.H, p.dk * p.dv, p.dk, p.n_min, p.H);
  CsTerms x = {nullptr, nullptr, nullptr};
  if (!MLSTM && tensor)
    x = {(uint8_t*)scratch + l.Xq, (uint8_t*)scratch + l.Xk, (unsigned long long*)(scratch + l.odd)};
  if (const int e = bf_launch_pdl(cs_qk_kernel<A, false>, dim3(l.chunks, p.QH, tiles * tiles + (x.q ? 2 : 0)),
                                  dim3(256), 0, stream, qk, p, q_start, qkm, (float*)nullptr, x))
    return e;
  if constexpr (MLSTM) {
    if (tensor)
      return mt_launch(qk, p, l.chunks, q_start, state, slot_stride, state_size, state_slots, n_slots, G, Hs, g0,
                       Wl, E, qkm, U, Un, o_raw, err, stream);
  } else if (tensor) {
    if (const int e = ct_configure()) return e;
    CtHead* W = (CtHead*)(scratch + l.W);
    ct_weights_kernel<<<dim3(l.chunks, p.H), 256, 0, stream>>>(p, q_start, G, Hs, g0, qkm, W);
    ct_state_kernel<<<dim3(p.dv / CT_SV * (p.dk / 128), p.H, p.B), CT_S_THREADS, CT_S_SMEM, stream>>>(
        qk, v, p, q_start, state, slot_stride, state_slots, n_slots, G, Wl, x.k, x.odd, U, err);
    ct_out_launch(qk, v, p, l.chunks, q_start, state_slots, n_slots, G, Hs, W, qkm, x.q, x.odd, U, o_raw, err, stream);
    return bf_launch_status();
  }
  cs_state_kernel<A, V, MLSTM><<<dim3(l.chunks, p.H, tk * tv), CS_THREADS, 0, stream>>>(
      qk, v, p, q_start, Wl, U, Un);
  const int elems = p.dk * p.dv + (MLSTM ? p.dk : 0);
  cs_prefix_kernel<MLSTM><<<dim3((elems + 511) / 512, p.H, p.B), 128, 0, stream>>>(
      state, slot_stride, state_size, state_slots, n_slots, p, q_start, G, g0, U, Un, err);
  cs_out_kernel<A, V, MLSTM, MLSTM><<<dim3(l.chunks, p.H, tiles * tv), CS_THREADS, 0, stream>>>(
      qk, v, p, q_start, state_slots, n_slots, G, Hs, g0, E, qkm, U, Un, o_raw);
  return bf_launch_status();
}

static bool cs_sizes_ok(const CsIn& p, const void* state, long long slot_stride,
                        const void* o_raw) {
  return p.T > 0 && p.B > 0 && p.B <= 65535 && p.H > 0 && p.H <= 65535 && p.QH > 0 &&
         p.n_min >= 0 && p.H % p.QH == 0 && p.dk > 0 && p.dv > 0 && p.dk % 4 == 0 && p.dv % 4 == 0 && p.C > 0 &&
         p.C % CS_T == 0 && p.qk_stride % 4 == 0 && p.v_stride % 4 == 0 && slot_stride % 4 == 0 &&
         (((uintptr_t)state | (uintptr_t)o_raw) & 15) == 0;
}

// qk [T][2][QH][dk] (q, then k), vf [T][H][dv], float; a decay per head or per (token, head).
// State and o_raw as in bf_linear_scan; requests of at most n_min tokens are left alone.  terms: `scratch` has
// the room for the products on the tensor cores (chunk_tensor.cuh), which then run there.
BF_EXPORT int bf_chunk_scan_linear(const float* qk, const float* vf, const float* decays,
                                   const float* tok_decay, float* state, long long slot_stride,
                                   const int* q_start, const int* state_slots, int n_slots,
                                   float* o_raw, void* scratch, int T, int B, int H, int QH,
                                   int dk, int dv, int C, int n_min, int terms, int* err,
                                   cudaStream_t stream) {
  CsIn p = {0, (long long)QH * dk, 0, 2LL * QH * dk, (long long)H * dv, H, QH, dk, dv, C, T, B,
            n_min, 1.f};
  if (!cs_sizes_ok(p, state, slot_stride, o_raw) || (!decays && !tok_decay) || !scratch ||
      (((uintptr_t)qk | (uintptr_t)vf) & 15) ||
      (terms && !ct_takes(H, QH, dk, dv, C, cs_most_chunks(T, B, C, n_min))))
    return (int)cudaErrorInvalidValue;
  return cs_launch<float, float, false>(qk, vf, p, decays, tok_decay, nullptr, state, slot_stride,
                                        dk * dv, q_start, state_slots, n_slots, o_raw,
                                        (char*)scratch, err, stream, terms);
}

// proj rows [q: H dk | k: H dk | v: H dv | ...] in bfloat16, gates and state as in bf_mlstm_scan; max_q and
// min_ctas: mlstm_tensor.cuh, mt_takes.
BF_EXPORT int bf_chunk_scan_mlstm(const void* proj, long long stride, const float* gates,
                                  float* state, long long slot_stride, int state_size,
                                  const int* q_start, const int* state_slots, int n_slots,
                                  float* o_raw, void* scratch, int T, int B, int H, int dk, int dv,
                                  float q_scale, int C, int n_min, int max_q, int min_ctas, int* err,
                                  cudaStream_t stream) {
  CsIn p = {0, (long long)H * dk, 2LL * H * dk, stride, stride, H, H, dk, dv, C, T, B, n_min,
            q_scale};
  if (!cs_sizes_ok(p, state, slot_stride, o_raw) || state_size % 4 || !gates || !scratch ||
      ((uintptr_t)proj & 7))
    return (int)cudaErrorInvalidValue;
  const __nv_bfloat16* x = (const __nv_bfloat16*)proj;
  return cs_launch<__nv_bfloat16, __nv_bfloat16, true>(
      x, x, p, nullptr, nullptr, gates, state, slot_stride, state_size, q_start, state_slots,
      n_slots, o_raw, (char*)scratch, err, stream,
      mt_takes(p, proj, cs_most_chunks(T, B, C, n_min), max_q, min_ctas));
}

// How many kernels bf_chunk_scan_mlstm launches: four on the tensor cores, five of multiply-adds.
BF_EXPORT int bf_chunk_scan_mlstm_kernels(const void* proj, long long stride, int T, int B, int H, int dk,
                                          int dv, int C, int n_min, int max_q, int min_ctas) {
  const CsIn p = {0, (long long)H * dk, 2LL * H * dk, stride, stride, H, H, dk, dv, C, T, B, n_min, 1.f};
  return mt_takes(p, proj, cs_most_chunks(T, B, C, n_min), max_q, min_ctas) ? 4 : 5;
}

// The gated delta rule.  Scratch: F (G and H are the same array), g0, Wl | qkm | kkm | W | Y |
// u | Sc.
struct DsLayout {
  size_t F, g0, Wl, qkm, kkm, W, Y, u, Sc, Xq, Xk, odd, Ww, Xw, odd_w, total;
  int chunks;
};
static DsLayout ds_layout(int T, int B, int H, int G, int dk, int dv, int n_min, bool terms) {
  DsLayout l;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += (bytes + 255) & ~(size_t)255;
    return here;
  };
  l.chunks = cs_most_chunks(T, B, DS_C, n_min);
  l.F = take((size_t)T * H * 8);
  l.g0 = take((size_t)B * H * 8);
  l.Wl = take((size_t)T * H * 8);
  l.qkm = take((size_t)l.chunks * G * DS_C * DS_C * 4);
  l.kkm = take((size_t)l.chunks * G * DS_C * DS_C * 4);
  l.W = take((size_t)l.chunks * H * DS_C * dk * 4);
  l.Y = take((size_t)l.chunks * H * DS_C * dv * 4);
  l.u = take((size_t)T * H * dv * 4);
  l.Sc = take((size_t)l.chunks * H * dk * dv * 4);
  l.Xq = take(terms ? ct_terms_bytes(l.chunks, G, dk) : 0);
  l.Xk = take(terms ? ct_terms_bytes(l.chunks, G, dk) : 0);
  l.Xw = take(terms ? ct_terms_bytes(l.chunks, H, dk) : 0);
  l.odd_w = take(terms ? (size_t)l.chunks * H * 8 : 0);
  l.odd = take(terms ? (size_t)l.chunks * G * 16 : 0);
  l.Ww = take(terms ? (size_t)l.chunks * H * sizeof(CtHead) : 0);
  l.total = at;
  return l;
}

// terms: as for bf_chunk_scan_scratch
BF_EXPORT long long bf_chunk_scan_delta_scratch(int T, int B, int H, int G, int dk, int dv,
                                                int n_min, int terms) {
  if (terms && !ct_takes(H, G, dk, dv, DS_C, cs_most_chunks(T, B, DS_C, n_min))) return 0;
  return (long long)ds_layout(T, B, H, G, dk, dv, n_min, terms).total;
}

// qkv, gates, state and o_raw as in bf_delta_scan (keys and values of at most 128, multiples of 4);
// requests of at most n_min tokens are left alone.
BF_EXPORT int bf_chunk_scan_delta(const float* qkv, const float* gates, float* state,
                                  long long slot_stride, const int* q_start,
                                  const int* state_slots, int n_slots, float* o_raw, void* scratch,
                                  int T, int B, int H, int G, int dk, int dv, int n_min, int terms,
                                  int* err, cudaStream_t stream) {
  const long long C = 2LL * G * dk + (long long)H * dv;
  if (T <= 0 || B <= 0 || B > 65535 || H <= 0 || H > 65535 || G <= 0 || H % G || dk <= 0 ||
      n_min < 0 || dv <= 0 || dk > DS_D || dv > DS_D || dk % 4 || dv % 4 || !scratch ||
      (((uintptr_t)qkv | (uintptr_t)o_raw) & 15) ||
      (terms && !ct_takes(H, G, dk, dv, DS_C, cs_most_chunks(T, B, DS_C, n_min))))
    return (int)cudaErrorInvalidValue;
  const DsLayout l = ds_layout(T, B, H, G, dk, dv, n_min, terms);
  char* base = (char*)scratch;
  double* F = (double*)(base + l.F);
  double* g0 = (double*)(base + l.g0);
  float2* Wl = (float2*)(base + l.Wl);
  float* qkm = (float*)(base + l.qkm);
  float* kkm = (float*)(base + l.kkm);
  float* W = (float*)(base + l.W);
  float* Y = (float*)(base + l.Y);
  float* u = (float*)(base + l.u);
  float* Sc = (float*)(base + l.Sc);
  uint8_t* Xq = terms ? (uint8_t*)base + l.Xq : nullptr;
  unsigned long long* odd = (unsigned long long*)(base + l.odd);
  CtHead* Ww = (CtHead*)(base + l.Ww);
  const DsIn d = {qkv, gates, C, H, G, dk, dv, T, B, n_min};
  // (the decays are the second rows of gates: [T][2][H])
  const CsIn p = {0, (long long)G * dk, 0, C, (long long)H * dv, H, G, dk, dv, DS_C, T, B, n_min,
                  1.f};
  const size_t smem_prep = ((size_t)2 * DS_C * DS_P + 2 * DS_C * 68 + 16 * 52) * sizeof(float);
  const size_t smem_walk = ((size_t)4 * DS_C * DS_P + (DS_D + DS_C) * (DS_NS + 4)) * sizeof(float);
  static bool configured[BF_MAX_DEVICES];
  bool& done = configured[bf_current_device()];
  if (!done) {
    cudaError_t e = cudaFuncSetAttribute(
        ds_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_prep);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ds_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem_walk);
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  if (terms) {
    if (const int e = ct_configure()) return e;
  }
  cs_gates_kernel<false><<<dim3(H, B), CS_GATE_THREADS, 0, stream>>>(
      nullptr, gates + H, nullptr, state, slot_stride, dk * dv, q_start, state_slots, n_slots, F, F,
      nullptr, g0, Wl, DS_C, T, H, dk * dv, dk, n_min, 2 * H);
  const CsTerms x = {Xq, terms ? (uint8_t*)base + l.Xk : nullptr, odd};
  uint8_t* Xw = terms ? (uint8_t*)base + l.Xw : nullptr;
  unsigned long long* odd_w = (unsigned long long*)(base + l.odd_w);
  if (const int e = bf_launch_pdl(cs_qk_kernel<float, true>, dim3(l.chunks, G, x.q ? 3 : 1), dim3(256), 0, stream,
                                  qkv, p, q_start, qkm, kkm, x))
    return e;
  ds_prep_kernel<<<dim3(l.chunks, H), DS_PREP_THREADS, smem_prep, stream>>>(d, q_start, F, kkm, W,
                                                                            Y, qkm, terms ? Ww : nullptr, Xw, odd_w);
  if (terms) {
    dt_walk_kernel<<<dim3(dv / CT_SV, H, B), DT_THREADS, DT_SMEM, stream>>>(
        d, q_start, state_slots, n_slots, state, slot_stride, F, Wl, W, Y, Xw, odd_w, x.k, odd, u, Sc, err);
    ct_out_launch(qkv, u, p, l.chunks, q_start, state_slots, n_slots, F, F, Ww, qkm, Xq, odd, Sc, o_raw, err, stream);
    return bf_launch_status();
  }
  ds_walk_kernel<<<dim3((dv + DS_NS - 1) / DS_NS, H, B), 128, smem_walk, stream>>>(
      d, q_start, state_slots, n_slots, state, slot_stride, F, Wl, W, Y, u, Sc, err);
  cs_out_kernel<float, float, false, true>
      <<<dim3(l.chunks, H, (dv + CS_T - 1) / CS_T), CS_THREADS, 0, stream>>>(
          qkv, u, p, q_start, state_slots, n_slots, F, F, g0, nullptr, qkm, Sc, nullptr, o_raw);
  return bf_launch_status();
}
