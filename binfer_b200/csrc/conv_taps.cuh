// The short causal convolution in front of several mixers, four neighbouring channels a thread over a
// run of consecutive tokens: a token's value enters registers once and serves all its taps.
//
//   y_t[c] = y0[c] + sum_j w[c, j] u_{t - taps + 1 + j}[c],   j = 0 .. taps-1, ascending
//
// Tokens whose taps reach behind the step's first row of their request read the request's state
// ([taps-1, C] floats, oldest first).  The kernels that walk tokens one warp at a time fetched every
// value `taps` times in pieces of two or four bytes a lane, which is what bounded them.
#pragma once
#include "common.cuh"

__device__ __forceinline__ float4 ct_ld4(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ float4 ct_ld4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void ct_st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void ct_st4(__nv_bfloat16* p, float4 v) {
  uint2 raw;
  *reinterpret_cast<__nv_bfloat162*>(&raw.x) = __floats2bfloat162_rn(v.x, v.y);
  *reinterpret_cast<__nv_bfloat162*>(&raw.y) = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = raw;
}
__device__ __forceinline__ float ct_silu(float y) { return y / (1.f + expf(-y)); }
__device__ __forceinline__ float4 ct_silu4(float4 y) {
  return make_float4(ct_silu(y.x), ct_silu(y.y), ct_silu(y.z), ct_silu(y.w));
}

// Whether weights and states can be read so (channels in fours).
static inline bool ct_aligned(const float* conv_w, const float* state, long long state_stride) {
  return ((((uintptr_t)conv_w | (uintptr_t)state) & 15) | (state_stride & 3)) == 0;
}

// Tokens of a run, for `units` threads of four channels a token: runs share fetches, but a step of
// few tokens needs its threads.
static inline int ct_run(long long T, long long units) {
  return T * units >= 148LL * 2048 * 8 ? 8 : T * units >= 148LL * 2048 * 2 ? 2 : 1;
}

template <int TAPS>
struct ConvTaps {
  float4 w[TAPS];
  float4 h[TAPS > 1 ? TAPS - 1 : 1];         // the values before the current one, oldest first

  __device__ __forceinline__ void weights(const float* __restrict__ conv_w, int c) {
    // four channels' taps side by side, in 16-byte pieces
    float v[4 * TAPS];
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {
      const float4 x = ct_ld4(conv_w + (size_t)c * TAPS + 4 * j);
      v[4 * j] = x.x;
      v[4 * j + 1] = x.y;
      v[4 * j + 2] = x.z;
      v[4 * j + 3] = x.w;
    }
#pragma unroll
    for (int j = 0; j < TAPS; ++j)
      w[j] = make_float4(v[j], v[TAPS + j], v[2 * TAPS + j], v[3 * TAPS + j]);
  }
  // the values before the request's token `local` of this step, whose row is `row`
  template <typename A>
  __device__ __forceinline__ void history(const A* row, long long stride, int c, int local,
                                          const float* __restrict__ st, int C) {
#pragma unroll
    for (int j = 0; j < TAPS - 1; ++j) {
      const int back = TAPS - 1 - j;
      if (local >= back) {
        h[j] = ct_ld4(row - (size_t)back * stride + c);
      } else {
        h[j] = ct_ld4(st + (size_t)(TAPS - 1 + local - back) * C + c);
      }
    }
  }
  __device__ __forceinline__ float4 step(float4 y, float4 u) {
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {
      const float4 v = j < TAPS - 1 ? h[j < TAPS - 1 ? j : 0] : u;
      y.x += w[j].x * v.x;
      y.y += w[j].y * v.y;
      y.z += w[j].z * v.z;
      y.w += w[j].w * v.w;
    }
#pragma unroll
    for (int j = 0; j + 1 < TAPS - 1; ++j) h[j] = h[j + 1];
    if (TAPS > 1) h[TAPS > 1 ? TAPS - 2 : 0] = u;
    return y;
  }
};

// The request of token t and the token's number among the request's tokens of this step; the state
// rows of that request (slot 0's, flagged, where the slot is none).
struct ConvPlace {
  int local;
  const float* st;
};
__device__ __forceinline__ ConvPlace ct_place(int t, const int* __restrict__ seq_of_token,
                                              const int* __restrict__ q_start,
                                              const int* __restrict__ state_slots,
                                              int n_state_slots, const float* __restrict__ state,
                                              long long state_stride, int taps,
                                              int* __restrict__ err) {
  ConvPlace p;
  const int b = seq_of_token[t];
  p.local = t - q_start[b];
  int slot = 0;
  if (taps > 1) {
    slot = state_slots[b];
    if (slot < 0 || slot >= n_state_slots) {
      atomicOr(err, BF_ERR_SLOT);
      slot = 0;
    }
  }
  p.st = state + (size_t)slot * state_stride;
  return p;
}
