// True 32-bit matrix product for the float32 engine: C[M,N] = A[M,K] * W[N,K]^T, for sums of
// fewer than 512 terms (longer ones: sgemm_split.cu), and for sums of any length where the float32 engine
// checks the tensor cores' paths and should share nothing with them (ops.sgemm_nt, multiply_adds).
//
// Plain FP32 FMAs on the CUDA cores; no tensor-core mode of any kind.
// The reference has no 32-bit product at all: every dense product is a cuBLAS
// bf16 call with float accumulation (cuda/kernels/gemm.cu:244-267); the operand
// layout here is the same (weights as stored, [out, in] row-major).
//
// Every output element is summed in one order that depends on K alone, whatever M,
// N or the tile variant, so a token's result does not depend on which other tokens
// share the batch: ascending runs of SG_RUN terms, one fmaf per term, and the runs'
// sums added in ascending order.  (One sequential sum has a rounding error that grows
// with sqrt(K): at the 12288 inner features of the Qwen3-8B shape it stood at 5e-6 of
// the logits' rms.  In runs of 64 it grows with sqrt(64 + K / 64).)
//
// What bounds it: the FP32 pipes (74 TFLOP/s nominal), and for few rows the bytes of W.  A step of
// 16 terms is fetched into registers while the one before is multiplied from shared memory (two
// buffers, one barrier a step), as 16-byte pieces of K where sizes, strides and addresses allow,
// else term by term.  The multiply-adds are packed pairs of rows (fma.rn.f32x2: both halves
// rounded on their own, so every sum is what single ones give): half the instructions, which
// leaves issue slots to the shared-memory reads (2,048 x 4,096 x 2,048: 802 us, 42.9 TFLOP/s,
// against 991 with single ones; 1,635 before, when each step was fetched, stored and only then
// multiplied; 333 rows: 394 -> 190 us; one row: 194 -> 53).  Tiles of 64 x 128 and 128 x 128
// with 8 x 8 outputs a thread: 880 and 955 us; steps of 32 terms: 888.
#include "common.cuh"

#define SG_RUN 64

__device__ __forceinline__ unsigned long long sg_pair(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void sg_unpair(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long sg_fma2(unsigned long long a, unsigned long long b,
                                                      unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long sg_add2(unsigned long long a,
                                                      unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// A thread's TM x TN outputs are TM / 2 pairs of rows.  VEC: K in whole pieces of four, every row
// of A and W on a 16-byte boundary.
template <int BM, int BN, int BK, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
sgemm_nt_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                int M, int N, int K, long long lda, long long ldw, long long ldc,
                long long batch_a, long long batch_w, long long batch_c) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  // pieces of four that a thread fetches (at BM 16 not every thread has one of A)
  constexpr int KP = BK / 4;
  constexpr int PA = (BM * KP + THREADS - 1) / THREADS, PW = BN * KP / THREADS;
  static_assert(TM % 2 == 0 && TN % 4 == 0, "pairs of rows, 16-byte reads of W's columns");
  static_assert((BM * KP % THREADS == 0 || PA == 1) && BN * KP % THREADS == 0, "whole pieces a thread");
  static_assert(SG_RUN % BK == 0, "a run is a whole number of K steps");
  A += blockIdx.z * batch_a;             // one product per blockIdx.z (strides 0: one product)
  W += blockIdx.z * batch_w;
  C += blockIdx.z * batch_c;
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Ws[2][BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  unsigned long long acc[TM / 2][TN], total[TM / 2][TN];   // the current run; the runs before it
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = total[i][j] = 0ull;

  float pa[PA][4], pw[PW][4];
  auto piece = [&](const float* base, int row, int rows, long long ld, int k, float (&x)[4]) {
    x[0] = x[1] = x[2] = x[3] = 0.f;
    if (row >= rows) return;
    const float* src = base + (size_t)row * ld + k;
    if (VEC) {
      if (k < K) {
        const float4 v = *reinterpret_cast<const float4*>(src);
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (k + e < K) x[e] = src[e];
    }
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int idx = tid + i * THREADS;
      if (idx < BM * KP) piece(A, m0 + idx / KP, M, lda, k0 + 4 * (idx % KP), pa[i]);
    }
#pragma unroll
    for (int i = 0; i < PW; ++i) {
      const int idx = tid + i * THREADS;
      piece(W, n0 + idx / KP, N, ldw, k0 + 4 * (idx % KP), pw[i]);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int idx = tid + i * THREADS;
      if (idx < BM * KP) {
#pragma unroll
        for (int e = 0; e < 4; ++e) As[buf][4 * (idx % KP) + e][idx / KP] = pa[i][e];
      }
    }
#pragma unroll
    for (int i = 0; i < PW; ++i) {
      const int idx = tid + i * THREADS;
#pragma unroll
      for (int e = 0; e < 4; ++e) Ws[buf][4 * (idx % KP) + e][idx / KP] = pw[i][e];
    }
  };
  fetch(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
    if (k0 + BK < K) fetch(k0 + BK);
    // A zero-filled tail (beyond K) adds +0 terms, which leave every sum unchanged.
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      unsigned long long a[TM / 2], b[TN];
      if (TM % 4 == 0) {
#pragma unroll
        for (int i = 0; i < TM / 4; ++i) {
          const ulonglong2 v =
              *reinterpret_cast<const ulonglong2*>(&As[buf][kk][ty * TM + 4 * i]);
          a[2 * i] = v.x;
          a[(2 * i + 1) % (TM / 2)] = v.y;
        }
      } else {
#pragma unroll
        for (int i = 0; i < TM / 2; ++i)
          a[i] = *reinterpret_cast<const unsigned long long*>(&As[buf][kk][ty * TM + 2 * i]);
      }
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const float4 w = *reinterpret_cast<const float4*>(&Ws[buf][kk][tx * 4 + j * (BN / TN * 4)]);
        b[4 * j] = sg_pair(w.x, w.x);
        b[4 * j + 1] = sg_pair(w.y, w.y);
        b[4 * j + 2] = sg_pair(w.z, w.z);
        b[4 * j + 3] = sg_pair(w.w, w.w);
      }
#pragma unroll
      for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = sg_fma2(a[i], b[j], acc[i][j]);
    }
    if ((k0 + BK) % SG_RUN == 0 || k0 + BK >= K) {   // a run ends (the last may be short)
#pragma unroll
      for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          total[i][j] = sg_add2(total[i][j], acc[i][j]);
          acc[i][j] = 0ull;
        }
    }
    if (k0 + BK < K) store(buf ^ 1);    // (read last before the barrier of the step before)
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM / 2; ++i) {
    const int gm = m0 + ty * TM + 2 * i;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * 4 + (j / 4) * (BN / TN * 4) + j % 4;
      float lo, hi;
      sg_unpair(total[i][j], lo, hi);
      if (gn < N && gm < M) C[(size_t)gm * ldc + gn] = lo;
      if (gn < N && gm + 1 < M) C[(size_t)(gm + 1) * ldc + gn] = hi;
    }
  }
}

template <int BM, int BN, int BK, int TM, int TN>
static void sgemm_go(const float* A, const float* W, float* C, int M, int N, int K, long long lda,
                     long long ldw, long long ldc, int batch, long long batch_a,
                     long long batch_w, long long batch_c, cudaStream_t stream) {
  constexpr int threads = (BM / TM) * (BN / TN), most = 65535 * BM;   // (rows of a launch)
  const bool vec = ((K | lda | ldw | batch_a | batch_w) & 3) == 0 &&
                   (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  for (int m0 = 0; m0 < M; m0 += most) {
    const int m = M - m0 < most ? M - m0 : most;
    const dim3 grid((N + BN - 1) / BN, (m + BM - 1) / BM, batch);
    const float* a = A + m0 * lda;
    float* c = C + m0 * ldc;
    if (vec)
      sgemm_nt_kernel<BM, BN, BK, TM, TN, true><<<grid, threads, 0, stream>>>(
          a, W, c, m, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
    else
      sgemm_nt_kernel<BM, BN, BK, TM, TN, false><<<grid, threads, 0, stream>>>(
          a, W, c, m, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
    if (M - m0 <= most) break;
  }
}

static int sgemm_nt_launch(const float* A, const float* W, float* C, int M, int N, int K,
                           long long lda, long long ldw, long long ldc, int batch,
                           long long batch_a, long long batch_w, long long batch_c,
                           cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  // Rows of a tile: 64, 32 or 16.  More rows a tile read W fewer times and keep the FP32 pipes
  // fuller (2,048 rows of 2,048 terms against 12,288 outputs: 44 TFLOP/s in tiles of 64, 31 in
  // tiles of 32, 17 in tiles of 16), but a grid that leaves SMs idle costs more: with n tiles on
  // the busiest SM a product of 2,048 terms took about 45 (n + 1), 30 + 33 n and 18 + 30 n us
  // (n from 1 to 4; 16 rows: 48, 77, 110, 145 us).  Take the shape whose line is lowest.
  const long long cols = (N + 63) / 64 * (long long)batch;
  auto busiest = [&](int rows) { return ((M + rows - 1) / rows * cols + 147) / 148; };
  const long long c64 = 45 + 45 * busiest(64), c32 = 30 + 33 * busiest(32),
                  c16 = 18 + 30 * busiest(16);
#define SG_GO(...)                                                                            \
  sgemm_go<__VA_ARGS__>(A, W, C, M, N, K, lda, ldw, ldc, batch, batch_a, batch_w, batch_c, stream)
  if (M <= 16 || (c16 <= c32 && c16 <= c64)) SG_GO(16, 64, 16, 2, 4);
  else if (c32 <= c64) SG_GO(32, 64, 32, 4, 4);
  else SG_GO(64, 64, 16, 8, 4);
#undef SG_GO
  return bf_launch_status();
}

BF_EXPORT int bf_sgemm_nt(const float* A, const float* W, float* C, int M, int N, int K,
                          long long lda, long long ldw, long long ldc, cudaStream_t stream) {
  return sgemm_nt_launch(A, W, C, M, N, K, lda, ldw, ldc, 1, 0, 0, 0, stream);
}

// `batch` products at once: product b reads A + b batch_a and W + b batch_w and writes
// C + b batch_c (heads that lie side by side in a token's row, each with a matrix of its own).
BF_EXPORT int bf_sgemm_nt_batched(const float* A, const float* W, float* C, int M, int N, int K,
                                  long long lda, long long ldw, long long ldc, int batch,
                                  long long batch_a, long long batch_w, long long batch_c,
                                  cudaStream_t stream) {
  if (batch > 65535) return (int)cudaErrorInvalidValue;
  return sgemm_nt_launch(A, W, C, M, N, K, lda, ldw, ldc, batch, batch_a, batch_w, batch_c,
                         stream);
}
