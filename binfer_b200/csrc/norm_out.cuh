// A head's output o over its root mean square, times a weight, times silu or sigmoid of a gate: one
// warp per (token, head), the head's numbers in registers (NV pieces of four a lane: NV * 128 numbers
// a head).  One pass over o where the kernels for any size take two, in 16-byte pieces:
// 2,000 tokens of 8 heads of 512 20 us there and 15 here, of 16 heads of 128 15.6 and 9.
//   out = o * rsqrt(mean o^2 + eps) * out_scale * w * act(gate)
#pragma once
#include "conv_taps.cuh"

template <typename A, int NV>
__global__ void __launch_bounds__(128) norm_out_vec_kernel(
    const float* __restrict__ o_raw, const A* __restrict__ proj, long long stride, long long g_off,
    const float* __restrict__ weight, long long w_head, int sigmoid, A* __restrict__ out,
    long long out_stride, long long items, int H, float eps, float out_scale) {
  const long long item = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (item >= items) return;
  const int lane = threadIdx.x & 31;
  const long long t = item / H;
  const int h = (int)(item % H);
  constexpr int dv = NV * 128;
  const float* o = o_raw + (size_t)item * dv + lane * 4;
  const A* g = proj + (size_t)t * stride + g_off + (size_t)h * dv + lane * 4;
  float4 v[NV], z[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = ct_ld4(o + 128 * i);
#pragma unroll
  for (int i = 0; i < NV; ++i) z[i] = ct_ld4(g + 128 * i);
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    ss += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
  const float f = rsqrtf(warp_sum(ss) / (float)dv + eps) * out_scale;
  A* dst = out + (size_t)t * out_stride + (size_t)h * dv + lane * 4;
  auto act = [&](float x) {
    const float s = 1.f / (1.f + expf(-x));
    return sigmoid ? s : x * s;
  };
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
    if (weight) w = ct_ld4(weight + (size_t)h * w_head + lane * 4 + 128 * i);
    ct_st4(dst + 128 * i,
           make_float4(v[i].x * f * w.x * act(z[i].x), v[i].y * f * w.y * act(z[i].y),
                       v[i].z * f * w.z * act(z[i].z), v[i].w * f * w.w * act(z[i].w)));
  }
}

// Launches it where the sizes and addresses are whole pieces of four; false, having done nothing,
// otherwise.  The choice does not depend on the number of tokens.  w_head: from one head's weights to
// the next one's (0: shared).
template <typename A>
static bool norm_out_vec(const float* o_raw, const A* proj, long long stride, long long g_off,
                         const float* weight, long long w_head, int sigmoid, A* out,
                         long long out_stride, int T, int H, int dv, float eps, float out_scale,
                         cudaStream_t stream) {
  const uintptr_t a = 4 * sizeof(A) - 1;
  if (((stride | g_off | out_stride | w_head) & 3) || (((uintptr_t)proj | (uintptr_t)out) & a) ||
      (((uintptr_t)o_raw | (uintptr_t)weight) & 15))
    return false;
  const long long items = (long long)T * H;
  const unsigned blocks = (unsigned)((items + 3) / 4);
#define NORM_OUT_GO(N)                                                                            \
  norm_out_vec_kernel<A, N><<<blocks, 128, 0, stream>>>(o_raw, proj, stride, g_off, weight, w_head, \
                                                        sigmoid, out, out_stride, items, H, eps,   \
                                                        out_scale)
  if (dv == 128) NORM_OUT_GO(1);
  else if (dv == 256) NORM_OUT_GO(2);
  else if (dv == 512) NORM_OUT_GO(4);
  else return false;
#undef NORM_OUT_GO
  return true;
}
