// A selective state space layer with a scalar decay per head and token (Mamba-2), around its
// recurrence, which the linear scan of retention.cu runs (bf_linear_scan: q = C, k = B,
// v = dt x, a decay per token and head):
//
//   S_t = exp(-exp(A_log_h) dt_t) S_{t-1} + dt_t B_t x_t^T      y_t = S_t^T C_t + D_h x_t
//
//   mamba2_encode   a row of `proj` holds [z: inner | x: inner | B: G N | C: G N | dt: H].  x, B
//                   and C (the channels from `xbc_off`) pass a causal convolution per channel
//                   with a bias and silu; the request's state (`state[slot]` = [taps-1, channels]
//                   of projected values, oldest first) lies behind the step's first row.  dt
//                   becomes softplus(dt + dt_bias_h).  Results, all float: qk [T][2][G][N] (C,
//                   then B), vf [T][H][P] = dt x, skip [T][H][P] = D_h x, decay [T][H].
//                   One warp per (token, head of x or group of B or of C).
//   gate_norm_out   y = (o_raw + skip) * silu(z), then an RMS norm in `parts` equal parts of
//                   the row (each by its own root mean square), times a weight per column.
//                   One block per (token, part).
//
// All arithmetic is float; only the projection's values and the result have the activation
// type.
#include "common.cuh"
#include "conv_taps.cuh"

#define M2_MAX_TAPS 16

__device__ __forceinline__ float m2_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

template <typename A>
__global__ void mamba2_encode_kernel(
    const A* __restrict__ proj, long long stride, long long xbc_off, long long dt_off,
    const float* __restrict__ conv_w, const float* __restrict__ conv_b, int taps,
    const float* __restrict__ state, long long state_stride, const int* __restrict__ state_slots,
    int n_state_slots, const int* __restrict__ seq_of_token, const int* __restrict__ q_start,
    const float* __restrict__ A_log, const float* __restrict__ dt_bias,
    const float* __restrict__ D, float* __restrict__ qk, float* __restrict__ vf,
    float* __restrict__ skip, float* __restrict__ decay, int T, int H, int G, int N, int P,
    int* __restrict__ err) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_token = H + 2 * G;
  const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
  if (item >= (long long)T * per_token) return;
  const int t = (int)(item / per_token), u = (int)(item % per_token);
  const int C = H * P + 2 * G * N;             // channels that pass the convolution
  int kind, d, c0;                             // 0 x, 1 B, 2 C; first channel of the unit
  if (u < H) { kind = 0; d = P; c0 = u * P; }
  else if (u < H + G) { kind = 1; d = N; c0 = H * P + (u - H) * N; }
  else { kind = 2; d = N; c0 = H * P + G * N + (u - H - G) * N; }
  const int b = seq_of_token[t];
  const int local = t - q_start[b];
  int slot = 0;
  if (taps > 1) {
    slot = state_slots[b];
    if (slot < 0 || slot >= n_state_slots) { atomicOr(err, BF_ERR_SLOT); slot = 0; }
  }
  const float* st = state + (size_t)slot * state_stride;
  const A* row = proj + (size_t)t * stride;
  float dt = 0.f, dskip = 0.f;
  if (kind == 0) {
    dt = m2_softplus(bf_ld(row + dt_off + u) + dt_bias[u]);
    dskip = D[u];
    if (lane == 0) decay[(size_t)t * H + u] = expf(-expf(A_log[u]) * dt);
  }
  for (int i = lane; i < d; i += 32) {
    const int c = c0 + i;
    float y = conv_b ? conv_b[c] : 0.f;
    if (taps >= 1) {
      for (int j = 0; j < taps; ++j) {
        const int src = local - (taps - 1) + j;
        const float v = src >= 0 ? bf_ld(proj + (size_t)(t - (taps - 1) + j) * stride + xbc_off + c)
                                 : st[(size_t)(taps - 1 + src) * C + c];
        y += conv_w[(size_t)c * taps + j] * v;
      }
    } else {
      y += bf_ld(row + xbc_off + c);
    }
    y = y / (1.f + expf(-y));
    if (kind == 0) {
      vf[((size_t)t * H + u) * P + i] = dt * y;
      skip[((size_t)t * H + u) * P + i] = dskip * y;
    } else if (kind == 1) {
      qk[(((size_t)t * 2 + 1) * G + (u - H)) * N + i] = y;          // k = B
    } else {
      qk[(((size_t)t * 2) * G + (u - H - G)) * N + i] = y;          // q = C
    }
  }
}

// The same, four channels a thread over a run of tokens (conv_taps.cuh), for heads and groups that
// are a multiple of four wide.  2,048 tokens of 4,096 + 2 x 1,024 channels, 4 taps: 40 us
// (bfloat16 in, float out), 112 with a warp per token; 256 tokens 10 and 16 (19 with the weights read
// number by number, a line of their own each).
template <typename A, int TAPS>
__global__ void __launch_bounds__(128) mamba2_encode_run_kernel(
    const A* __restrict__ proj, long long stride, long long xbc_off, long long dt_off,
    const float* __restrict__ conv_w, const float* __restrict__ conv_b,
    const float* __restrict__ state, long long state_stride, const int* __restrict__ state_slots,
    int n_state_slots, const int* __restrict__ seq_of_token, const int* __restrict__ q_start,
    const float* __restrict__ A_log, const float* __restrict__ dt_bias,
    const float* __restrict__ D, float* __restrict__ qk, float* __restrict__ vf,
    float* __restrict__ skip, float* __restrict__ decay, int T, int H, int G, int N, int P,
    int run, int* __restrict__ err) {
  const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
  const int X = H * P, C = X + 2 * G * N;
  if (c >= C) return;
  const int ta = blockIdx.y * run, tb = min(T, ta + run);
  const int head = c < X ? c / P : 0;
  float rate = 0.f, bias_dt = 0.f, d_skip = 0.f;
  if (c < X) {
    rate = -expf(A_log[head]);
    bias_dt = dt_bias[head];
    d_skip = D[head];
  }
  const float4 b4 = conv_b ? make_float4(conv_b[c], conv_b[c + 1], conv_b[c + 2], conv_b[c + 3])
                           : make_float4(0.f, 0.f, 0.f, 0.f);
  ConvTaps<TAPS> conv;
  conv.weights(conv_w, c);
  for (int t = ta; t < tb; ++t) {
    const A* row = proj + (size_t)t * stride;
    const ConvPlace at = ct_place(t, seq_of_token, q_start, state_slots, n_state_slots, state,
                                  state_stride, TAPS, err);
    if (t == ta || at.local == 0) conv.history(row + xbc_off, stride, c, at.local, at.st, C);
    const float4 y = ct_silu4(conv.step(b4, ct_ld4(row + xbc_off + c)));
    if (c < X) {
      const float dt = m2_softplus(bf_ld(row + dt_off + head) + bias_dt);
      if (c % P == 0) decay[(size_t)t * H + head] = expf(rate * dt);
      ct_st4(vf + (size_t)t * X + c, make_float4(dt * y.x, dt * y.y, dt * y.z, dt * y.w));
      ct_st4(skip + (size_t)t * X + c,
             make_float4(d_skip * y.x, d_skip * y.y, d_skip * y.z, d_skip * y.w));
    } else if (c < X + G * N) {
      ct_st4(qk + ((size_t)t * 2 + 1) * G * N + (c - X), y);            // k = B
    } else {
      ct_st4(qk + (size_t)t * 2 * G * N + (c - X - G * N), y);          // q = C
    }
  }
}

template <typename A>
static bool mamba2_encode_run(const A* proj, long long stride, long long xbc_off, long long dt_off,
                              const float* conv_w, const float* conv_b, int taps,
                              const float* state, long long state_stride, const int* state_slots,
                              int n_state_slots, const int* seq_of_token, const int* q_start,
                              const float* A_log, const float* dt_bias, const float* D, float* qk,
                              float* vf, float* skip, float* decay, int T, int H, int G, int N,
                              int P, int* err, cudaStream_t stream) {
  if (taps < 1 || taps > 4 || !ct_aligned(conv_w, state, state_stride) || P % 4 || N % 4 || stride % 4 || xbc_off % 4 ||
      ((uintptr_t)proj & (4 * sizeof(A) - 1)) ||
      (((uintptr_t)qk | (uintptr_t)vf | (uintptr_t)skip) & 15))
    return false;
  const int units = (H * P + 2 * G * N) / 4, run = ct_run(T, units);
  const dim3 grid((units + 127) / 128, (T + run - 1) / run);
  if (grid.y > 65535) return false;
#define M2_RUN(K)                                                                             \
  mamba2_encode_run_kernel<A, K><<<grid, 128, 0, stream>>>(                                   \
      proj, stride, xbc_off, dt_off, conv_w, conv_b, state, state_stride, state_slots,        \
      n_state_slots, seq_of_token, q_start, A_log, dt_bias, D, qk, vf, skip, decay, T, H, G, N, P, \
      run, err)
  if (taps == 1) M2_RUN(1);
  else if (taps == 2) M2_RUN(2);
  else if (taps == 3) M2_RUN(3);
  else M2_RUN(4);
#undef M2_RUN
  return true;
}

BF_EXPORT int bf_mamba2_encode(const void* proj, long long stride, long long xbc_off,
                               long long dt_off, const float* conv_w, const float* conv_b,
                               int taps, const float* state, long long state_stride,
                               const int* state_slots, int n_state_slots,
                               const int* seq_of_token, const int* q_start, const float* A_log,
                               const float* dt_bias, const float* D, float* qk, float* vf,
                               float* skip, float* decay, int T, int H, int G, int N, int P,
                               int act_dtype, int* err, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (taps > M2_MAX_TAPS || (taps > 1 && !state) || (taps >= 1 && !conv_w) || G <= 0 || H % G)
    return (int)cudaErrorInvalidValue;
  if (act_dtype == BF_DTYPE_F32
          ? mamba2_encode_run<float>((const float*)proj, stride, xbc_off, dt_off, conv_w, conv_b,
                                     taps, state, state_stride, state_slots, n_state_slots,
                                     seq_of_token, q_start, A_log, dt_bias, D, qk, vf, skip, decay,
                                     T, H, G, N, P, err, stream)
          : mamba2_encode_run<__nv_bfloat16>(
                (const __nv_bfloat16*)proj, stride, xbc_off, dt_off, conv_w, conv_b, taps, state,
                state_stride, state_slots, n_state_slots, seq_of_token, q_start, A_log, dt_bias, D,
                qk, vf, skip, decay, T, H, G, N, P, err, stream))
    return bf_launch_status();
  const int warps = 4;
  const long long items = (long long)T * (H + 2 * G);
  const unsigned blocks = (unsigned)((items + warps - 1) / warps);
  if (act_dtype == BF_DTYPE_F32)
    mamba2_encode_kernel<float><<<blocks, warps * 32, 0, stream>>>(
        (const float*)proj, stride, xbc_off, dt_off, conv_w, conv_b, taps, state, state_stride,
        state_slots, n_state_slots, seq_of_token, q_start, A_log, dt_bias, D, qk, vf, skip, decay,
        T, H, G, N, P, err);
  else
    mamba2_encode_kernel<__nv_bfloat16><<<blocks, warps * 32, 0, stream>>>(
        (const __nv_bfloat16*)proj, stride, xbc_off, dt_off, conv_w, conv_b, taps, state,
        state_stride, state_slots, n_state_slots, seq_of_token, q_start, A_log, dt_bias, D, qk,
        vf, skip, decay, T, H, G, N, P, err);
  return bf_launch_status();
}

// ------------------------------------------------------------------ gate_norm_out
// out[t, c] = y[c] * rsqrt(mean of y^2 over c's part + eps) * weight[c] with
// y[c] = (o_raw[t, c] + skip[t, c]) * silu(z[t, c]); the row has `parts` equal parts.
template <typename A>
__global__ void gate_norm_out_kernel(const float* __restrict__ o_raw,
                                     const float* __restrict__ skip, const A* __restrict__ proj,
                                     long long stride, long long z_off,
                                     const float* __restrict__ weight, A* __restrict__ out,
                                     long long out_stride, int n, int parts, float eps) {
  __shared__ float scratch[33];
  const int t = blockIdx.x, part = blockIdx.y;
  const int per = n / parts, c0 = part * per;
  const float* o = o_raw + (size_t)t * n + c0;
  const float* sk = skip ? skip + (size_t)t * n + c0 : nullptr;
  const A* z = proj + (size_t)t * stride + z_off + c0;
  A* dst = out + (size_t)t * out_stride + c0;
  float ss = 0.f;
  for (int i = threadIdx.x; i < per; i += blockDim.x) {
    const float g = bf_ld(z + i);
    const float y = (o[i] + (sk ? sk[i] : 0.f)) * (g / (1.f + expf(-g)));
    ss += y * y;
  }
  const float f = rsqrtf(block_sum(ss, scratch) / (float)per + eps);
  for (int i = threadIdx.x; i < per; i += blockDim.x) {
    const float g = bf_ld(z + i);
    const float y = (o[i] + (sk ? sk[i] : 0.f)) * (g / (1.f + expf(-g)));
    bf_st(dst + i, y * f * (weight ? weight[c0 + i] : 1.f));
  }
}

// The same with a warp per (token, part) and the part's numbers in registers (NV pieces of four a lane:
// parts of NV * 128 numbers): one pass, where the kernel above reads everything and takes every
// exponential twice.  2,008 rows of 4,096 in 8 parts: 20 us, 42 there.
template <typename A, int NV>
__global__ void __launch_bounds__(128) gate_norm_out_vec_kernel(
    const float* __restrict__ o_raw, const float* __restrict__ skip, const A* __restrict__ proj,
    long long stride, long long z_off, const float* __restrict__ weight, A* __restrict__ out,
    long long out_stride, long long items, int parts, float eps) {
  const long long item = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= items) return;
  const int lane = threadIdx.x & 31;
  const long long t = item / parts;
  const int c0 = (int)(item % parts) * NV * 128 + lane * 4;
  const size_t at = (size_t)t * parts * NV * 128 + c0;
  const A* z = proj + (size_t)t * stride + z_off + c0;
  float4 y[NV];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    y[i] = ct_ld4(o_raw + at + 128 * i);
    if (skip) {
      const float4 s = ct_ld4(skip + at + 128 * i);
      y[i] = make_float4(y[i].x + s.x, y[i].y + s.y, y[i].z + s.z, y[i].w + s.w);
    }
    const float4 g = ct_silu4(ct_ld4(z + 128 * i));
    y[i] = make_float4(y[i].x * g.x, y[i].y * g.y, y[i].z * g.z, y[i].w * g.w);
    ss += (y[i].x * y[i].x + y[i].y * y[i].y) + (y[i].z * y[i].z + y[i].w * y[i].w);
  }
  const float f = rsqrtf(warp_sum(ss) / (float)(NV * 128) + eps);
  A* dst = out + (size_t)t * out_stride + c0;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
    if (weight) w = ct_ld4(weight + c0 + 128 * i);
    ct_st4(dst + 128 * i, make_float4(y[i].x * f * w.x, y[i].y * f * w.y, y[i].z * f * w.z,
                                      y[i].w * f * w.w));
  }
}

template <typename A>
static bool gate_norm_out_vec(const float* o_raw, const float* skip, const A* proj, long long stride,
                              long long z_off, const float* weight, A* out, long long out_stride,
                              int T, int n, int parts, float eps, cudaStream_t stream) {
  const uintptr_t a = 4 * sizeof(A) - 1;
  if (((stride | z_off | out_stride) & 3) || (((uintptr_t)proj | (uintptr_t)out) & a) ||
      (((uintptr_t)o_raw | (uintptr_t)skip | (uintptr_t)weight) & 15))
    return false;
  const long long items = (long long)T * parts;
  const unsigned blocks = (unsigned)((items + 3) / 4);
#define GNO(N)                                                                                    \
  gate_norm_out_vec_kernel<A, N><<<blocks, 128, 0, stream>>>(                                     \
      o_raw, skip, proj, stride, z_off, weight, out, out_stride, items, parts, eps)
  const int per = n / parts;
  if (per == 128) GNO(1);
  else if (per == 256) GNO(2);
  else if (per == 512) GNO(4);
  else if (per == 1024) GNO(8);
  else return false;
#undef GNO
  return true;
}

BF_EXPORT int bf_gate_norm_out(const float* o_raw, const float* skip, const void* proj,
                               long long stride, long long z_off, const float* weight, void* out,
                               long long out_stride, int T, int n, int parts, float eps,
                               int act_dtype, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (parts <= 0 || n % parts) return (int)cudaErrorInvalidValue;
  if (act_dtype == BF_DTYPE_F32
          ? gate_norm_out_vec<float>(o_raw, skip, (const float*)proj, stride, z_off, weight,
                                     (float*)out, out_stride, T, n, parts, eps, stream)
          : gate_norm_out_vec<__nv_bfloat16>(o_raw, skip, (const __nv_bfloat16*)proj, stride, z_off,
                                             weight, (__nv_bfloat16*)out, out_stride, T, n, parts,
                                             eps, stream))
    return bf_launch_status();
  const int per = n / parts;
  const int threads = per > 1024 ? 256 : (per > 64 ? 128 : 32);
  dim3 grid(T, parts);
  if (act_dtype == BF_DTYPE_F32)
    gate_norm_out_kernel<float><<<grid, threads, 0, stream>>>(
        o_raw, skip, (const float*)proj, stride, z_off, weight, (float*)out, out_stride, n, parts,
        eps);
  else
    gate_norm_out_kernel<__nv_bfloat16><<<grid, threads, 0, stream>>>(
        o_raw, skip, (const __nv_bfloat16*)proj, stride, z_off, weight, (__nv_bfloat16*)out,
        out_stride, n, parts, eps);
  return bf_launch_status();
}
