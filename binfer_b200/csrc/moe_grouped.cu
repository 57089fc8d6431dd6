// A mixture's feed-forward for many tokens, each token through its chosen experts alone.
//
// The stacked product (gemm_tcgen05_pair.cu with a mixture) computes every expert for every token:
// E x T rows where top x T are wanted.  Here the tokens' rows are copied expert by expert, each
// expert's rows padded to tiles of 256, and two products on pairs of SMs walk those tiles, each
// against its expert's rows (or columns) of the stacked weights; the shared expert's tiles run in
// the same launches, on all tokens.
//
//   moe_sort      one block: the place of every (token, choice) in the sorted rows, in the tokens'
//                 order inside an expert; the expert of every tile; the rows' weights
//   moe_gather    the tokens' rows to their places
//   experts_pair<false>   gate and up projections, the activation and the weight in the epilogue
//   experts_pair<true>    down projections, float
//   moe_combine   a token's results added up in float: the shared expert's, then the choices' in the
//                 router's order, then the identity experts' share
//
// Identity choices (ids from E on) have no row.  A token's result depends on its own choices only:
// the sums of a row have one order whatever tile it lies in.
//
// The products' kernel is that of gemm_tcgen05_pair.cu: clusters of two CTAs on tiles of 256 rows x
// 256 accumulator columns (tcgen05.mma.cta_group::2), TMA both ways, two accumulators; what differs
// is where a tile's operands come from.  No load uses multicast; every wait is bounded.
//
// 2,048 tokens of width 2,048, 2 of 8 experts of 1,536 and a shared one: products 82 + 43 us, sort 8,
// gather 5, combine 9; the stacked products took 167 + 82.  What bounds it: the tensor pipe and, at
// this size, the last wave of tiles (256 rows an expert at least: up to E half-empty tiles).
#include <cuda.h>
#include <stdint.h>

#include "common.cuh"
#include "gate_act.cuh"
#include "pair_utils.cuh"
#include "tma_utils.cuh"
#include "umma_utils.cuh"

#define MG_TILE 256
#define MG_MAX_EXPERTS 64

// ------------------------------------------------------------------------------- moe_sort
// slot_of [T * top]: a row of the sorted buffer, -1 for an identity choice; row_w [rows]; meta[0]: the
// number of tiles, meta[1 + i]: tile i's expert.
__global__ void __launch_bounds__(1024) moe_sort_kernel(const int* __restrict__ top_ids,
                                                        const float* __restrict__ top_w, int n,
                                                        int E, int max_tiles,
                                                        int* __restrict__ slot_of,
                                                        float* __restrict__ row_w,
                                                        int* __restrict__ meta) {
  __shared__ int next[MG_MAX_EXPERTS];             // the expert's next free row
  __shared__ int warp_n[32][MG_MAX_EXPERTS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < MG_MAX_EXPERTS) next[tid] = 0;
  __syncthreads();
  for (int i = tid; i < n; i += 1024) {
    const int e = top_ids[i];
    if (e >= 0 && e < E) atomicAdd(next + e, 1);
  }
  __syncthreads();
  if (tid == 0) {
    int tiles = 0;
    for (int e = 0; e < E; ++e) {
      const int t = (next[e] + MG_TILE - 1) / MG_TILE;
      next[e] = tiles * MG_TILE;
      for (int i = 0; i < t && tiles + i < max_tiles; ++i) meta[1 + tiles + i] = e;
      tiles += t;
    }
    meta[0] = tiles < max_tiles ? tiles : max_tiles;   // (never more: max_tiles is n / 256 + E)
  }
  __syncthreads();
  for (int i0 = 0; i0 < n; i0 += 1024) {
    const int i = i0 + tid;
    int e = i < n ? top_ids[i] : -1;
    if (e < 0 || e >= E) e = -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int rank = __popc(same & ((1u << lane) - 1u));
    for (int x = lane; x < E; x += 32) warp_n[warp][x] = 0;
    __syncwarp();
    if (e >= 0 && rank == 0) warp_n[warp][e] = __popc(same);
    __syncthreads();
    if (tid < E) {                                 // the warps' counts to their first rows
      int at = next[tid];
      for (int w = 0; w < 32; ++w) {
        const int c = warp_n[w][tid];
        warp_n[w][tid] = at;
        at += c;
      }
      next[tid] = at;
    }
    __syncthreads();
    if (i < n) {
      const int slot = e >= 0 ? warp_n[warp][e] + rank : -1;
      slot_of[i] = slot;
      if (slot >= 0) row_w[slot] = top_w[i];
    }
    __syncthreads();
  }
}

// A warp per (token, choice): the token's row to its place.
__global__ void moe_gather_kernel(const __nv_bfloat16* __restrict__ x, long long stride,
                                  const int* __restrict__ slot_of, int n, int top, int width,
                                  __nv_bfloat16* __restrict__ xs) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) return;
  const int slot = slot_of[i];
  if (slot < 0) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(i / top) * stride);
  uint4* dst = reinterpret_cast<uint4*>(xs + (size_t)slot * width);
#pragma unroll 4
  for (int c = lane; c < width / 8; c += 32) dst[c] = src[c];
}

// Eight columns a thread: out[t] = bf16(y_sh[t] + sum_k y[slot_of[t, k]] + idw x[t]).
__global__ void moe_combine_kernel(const float* __restrict__ y, const float* __restrict__ y_sh,
                                   const int* __restrict__ slot_of, int T, int top, int width,
                                   const __nv_bfloat16* __restrict__ x, long long x_stride,
                                   const float* __restrict__ route_w, int rw_cols, int id_col,
                                   __nv_bfloat16* __restrict__ out) {
  const int w8 = width / 8;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)T * w8) return;
  const int t = (int)(i / w8), c = (int)(i % w8) * 8;
  float a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = 0.f;
  auto add = [&](const float* row) {
    const float4 p = *reinterpret_cast<const float4*>(row + c);
    const float4 q = *reinterpret_cast<const float4*>(row + c + 4);
    a[0] += p.x; a[1] += p.y; a[2] += p.z; a[3] += p.w;
    a[4] += q.x; a[5] += q.y; a[6] += q.z; a[7] += q.w;
  };
  if (y_sh) add(y_sh + (size_t)t * width);
  for (int k = 0; k < top; ++k) {
    const int slot = slot_of[(size_t)t * top + k];
    if (slot >= 0) add(y + (size_t)slot * width);
  }
  if (id_col >= 0) {
    const float w = route_w[(size_t)t * rw_cols + id_col];
    if (w != 0.f) {
      const uint4 raw = *reinterpret_cast<const uint4*>(x + (size_t)t * x_stride + c);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        a[2 * j] += w * f.x;
        a[2 * j + 1] += w * f.y;
      }
    }
  }
  uint4 o;
  __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(a[2 * j], a[2 * j + 1]);
  *reinterpret_cast<uint4*>(out + (size_t)t * width + c) = o;
}

namespace {

constexpr int EX_A_BYTES = 128 * BK * 2;      // a CTA's rows of one K slice
constexpr int EX_B_BYTES = 128 * BK * 2;      // ... and its half of the 256 weight rows
constexpr int EX_STAGE = EX_A_BYTES + EX_B_BYTES;
constexpr int EX_STAGES = 6;
constexpr int EX_OUT = 128 * 128;             // a staged slab: 128 rows of 128 bytes
constexpr int EX_BARS = 1024;
constexpr int EX_THREADS = 192;

struct ExpertsParams {
  int tokens, width, E, ff, ff_sh, F;
  int rows;                    // of the sorted buffers
  const int* meta;             // moe_sort's
  const float* row_w;          // [rows]
  const float* sh_w;           // the shared expert's weight per token (null: 1) ...
  int sh_w_stride;             // ... this many apart
  int clamped;                 // the activation: 0 silu, 1 clamped
  BfGateConst gk, gk_sh;
  int* err;
};

// A tile of a launch: the shared expert's first, then the sorted rows', rows fastest (pairs that work
// side by side read the same weights).
struct ExpertsTile {
  bool shared;
  int tt, tf, expert;
};

// DOWN false: rows [., width] x gate and up rows of the stacked [2 F, width] weight -> activations;
// DOWN true: activations x the expert's columns of the [width, F] weight -> float rows [., width].
template <bool DOWN>
__global__ void __launch_bounds__(EX_THREADS, 1)
experts_pair_kernel(const __grid_constant__ CUtensorMap map_a,      // sorted rows
                    const __grid_constant__ CUtensorMap map_a_sh,   // the shared expert's rows
                    const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ CUtensorMap map_out,
                    const __grid_constant__ CUtensorMap map_out_sh, const ExpertsParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(base);       // waited on in the leader only
  uint64_t* empty = full + EX_STAGES;
  uint64_t* acc_full = empty + EX_STAGES;                   // [2]
  uint64_t* acc_empty = acc_full + 2;                       // [2], waited on in the leader only
  uint64_t* drain = acc_empty + 2;                          // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* out_stage = base + EX_BARS;                      // [2] slabs on their way out
  uint8_t* tiles = out_stage + 2 * EX_OUT;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = pair_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int n_tiles = p.meta[0];
  const int tiles_sh = p.ff_sh ? (p.tokens + MG_TILE - 1) / MG_TILE : 0;
  const int cols = DOWN ? 256 : 128;                        // outputs of a tile
  const int tf_r = ((DOWN ? p.width : p.ff) + cols - 1) / cols;
  const int tf_s = ((DOWN ? p.width : p.ff_sh) + cols - 1) / cols;
  const int units_sh = tiles_sh * tf_s, units = units_sh + n_tiles * tf_r;
  auto tile_of = [&](int u) {
    ExpertsTile t;
    t.shared = u < units_sh;
    const int v = t.shared ? u : u - units_sh, m = t.shared ? tiles_sh : n_tiles;
    t.tt = v % m;
    t.tf = v / m;
    t.expert = t.shared ? p.E : p.meta[1 + t.tt];
    return t;
  };
  auto k_steps = [&](bool shared) {
    const int K = DOWN ? (shared ? p.ff_sh : p.ff) : p.width;
    return (K + BK - 1) / BK;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < EX_STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(acc_full + a, 1);
      mbar_init(acc_empty + a, 8);           // one arrival per epilogue warp of both CTAs
    }
    mbar_init(drain, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  pair_sync();                               // the peer's barriers exist before anything lands
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  int next = 0;                                // (copying thread) the stage behind its last fill
  uint32_t next_phase = 0;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      const uint32_t full_leader = pair_map(smem_u32(full), 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = pair; u < units && ok && !*abort; u += pairs) {
        const ExpertsTile t = tile_of(u);
        const int row = t.tt * MG_TILE + (int)rank * 128, first = t.expert * p.ff;
        const int steps = k_steps(t.shared);
        for (int kc = 0; kc < steps; ++kc) {
          if (!mbar_wait(empty + stage, phase ^ 1, abort)) {
            ok = false;
            break;
          }
          uint8_t* dst = tiles + (size_t)stage * EX_STAGE;
          const uint32_t bar = full_leader + 8u * (uint32_t)stage;
          if (rank == 0) mbar_expect_tx(full + stage, 2u * (uint32_t)EX_STAGE);
          pair_tma_load(dst, t.shared ? &map_a_sh : &map_a, bar, kc * BK, row);
          if (DOWN) {
            pair_tma_load(dst + EX_A_BYTES, &map_w, bar, first + kc * BK,
                          t.tf * 256 + (int)rank * 128);
          } else {
            // this CTA's columns: gate rows of 64 outputs, then the up rows of the same
            const int o0 = first + t.tf * 128 + (int)rank * 64;
            pair_tma_load(dst + EX_A_BYTES, &map_w, bar, kc * BK, o0);
            pair_tma_load(dst + EX_A_BYTES + 64 * BK * 2, &map_w, bar, kc * BK, p.F + o0);
          }
          if (++stage == EX_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      next = stage;
      next_phase = phase;
      // every arrival that the leader's commits send to this CTA's barriers lands before it ends
      for (int s = 0; s < EX_STAGES && ok && !*abort; ++s) {
        ok = mbar_wait(empty + stage, phase ^ 1, abort);
        if (++stage == EX_STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------- MMA issuer
    if (rank == 0) {
      // c = float, a = b = bf16, both K-major, N = 256, M = 256 over the pair
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) |
                             ((uint32_t)(MG_TILE >> 4) << 24);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int u = pair; u < units; u += pairs) {
        const int steps = k_steps(u < units_sh);
        if (!mbar_wait_warp(acc_empty + acc, acc_phase ^ 1, abort)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * 256);
        bool ok = true;
        for (int kc = 0; kc < steps; ++kc) {
          if (!mbar_wait_warp(full + stage, phase, abort)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(tiles + (size_t)stage * EX_STAGE);
          const uint64_t a_desc = umma_desc_k_sw128(a_addr);
          const uint64_t b_desc = umma_desc_k_sw128(a_addr + EX_A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            pair_umma(d_tmem, a_desc + (uint64_t)(2 * k), b_desc + (uint64_t)(2 * k), idesc,
                      (kc > 0 || k > 0) ? 1u : 0u);
          pair_commit_both(empty + stage);     // both CTAs' producers may refill the stage
          if (++stage == EX_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        pair_commit_both(acc_full + acc);      // both CTAs' epilogues may read the accumulator
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else {
    // --------------------------------------------------------------- epilogue
    const int quarter = warp & 3;              // the TMEM lanes this warp may read
    const uint32_t acc_empty_leader = pair_map(smem_u32(acc_empty), 0);
    int acc = 0;
    uint32_t acc_phase = 0;
    int n_stored = 0;                          // slabs handed to TMA stores so far
    for (int u = pair; u < units; u += pairs) {
      const ExpertsTile t = tile_of(u);
      const bool ok = !*abort && mbar_wait(acc_full + acc, acc_phase, abort);
      if (!epilogue_all(ok)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * 256);
      const int row = quarter * 32 + lane;     // of this CTA's 128
      const int y0 = t.tt * MG_TILE + (int)rank * 128;
      const int limit_y = t.shared ? p.tokens : p.rows;
      const int limit_x = DOWN ? p.width : t.shared ? p.ff_sh : p.ff;
      float wgt = 1.f;
      BfGateConst k = p.gk;
      if (!DOWN) {
        if (t.shared) {
          k = p.gk_sh;
          if (p.sh_w) wgt = p.sh_w[(size_t)min(y0 + row, p.tokens - 1) * p.sh_w_stride];
        } else {
          wgt = p.row_w[y0 + row];
        }
      }
      const int slabs = DOWN ? 8 : 2;
      for (int slab = 0; slab < slabs; ++slab) {
        uint8_t* buf = out_stage + (n_stored & 1) * EX_OUT;
        if (threadIdx.x == 64) bf_bulk_wait_read<1>();   // the store before last has read it
        epilogue_sync();
        if (DOWN) {
          uint32_t r[32];
          tmem_ld32(taddr + slab * 32, r);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            *reinterpret_cast<uint4*>(buf + row * 128 + ((q ^ (row & 7)) << 4)) =
                make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
        } else {
#pragma unroll
          for (int hs = 0; hs < 2; ++hs) {
            uint32_t r[32], up[32];
            tmem_ld32(taddr + slab * 128 + hs * 32, r);
            tmem_ld32(taddr + slab * 128 + hs * 32 + 64, up);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float g = __uint_as_float(r[j]), uu = __uint_as_float(up[j]);
              r[j] = __float_as_uint(wgt * (p.clamped ? bf_gate_mul_fast<BF_ACT_CLAMPED>(g, uu, k)
                                                      : bf_gate_mul_fast<BF_ACT_SILU>(g, uu, k)));
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 v;
              v.x = pack_bf16x2(r[8 * q], r[8 * q + 1]);
              v.y = pack_bf16x2(r[8 * q + 2], r[8 * q + 3]);
              v.z = pack_bf16x2(r[8 * q + 4], r[8 * q + 5]);
              v.w = pack_bf16x2(r[8 * q + 6], r[8 * q + 7]);
              const int chunk = hs * 4 + q;
              *reinterpret_cast<uint4*>(buf + row * 128 + ((chunk ^ (row & 7)) << 4)) = v;
            }
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        epilogue_sync();
        if (threadIdx.x == 64) {
          const int x = DOWN ? t.tf * 256 + slab * 32 : t.tf * 128 + slab * 64;
          if (x < limit_x && y0 < limit_y)
            bf_tma_store_2d(t.shared ? &map_out_sh : &map_out, buf, x, y0);
          bf_bulk_commit();
        }
        ++n_stored;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair_arrive_remote(acc_empty_leader + 8u * (uint32_t)acc);
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (threadIdx.x == 64) bf_bulk_wait_read<0>();   // shared memory stays until the stores read it
  }

  // ------------------------------------------------------------------ wind-down
  __syncthreads();
  if (*abort) {
    if (threadIdx.x == 0) {
      atomicOr(p.err, BF_ERR_WAIT);
      // the peer leaves its waits at once instead of running each of them out
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(
                       pair_map(smem_u32(const_cast<int*>(abort)), rank ^ 1u)),
                   "r"(1)
                   : "memory");
    }
    if (warp == 0 && lane == 0 && rank == 0) {
      mbar_drain(full, EX_STAGES, next, next_phase);  // copies that were issued but never consumed
    }
    if (warp == 1 && rank == 0) {
      pair_commit_own(drain);                  // products still in flight
      const long long t0 = clock64();
      while (!mbar_try_wait(drain, 0) && clock64() - t0 < WAIT_LIMIT_CYCLES / 16) {
      }
    }
    __syncthreads();
  }
  tc_fence_before();
  pair_sync();                                 // neither CTA's memory goes while the other uses it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(512)
                 : "memory");
  }
}

template <bool DOWN>
int experts_launch(const CUtensorMap& a, const CUtensorMap& a_sh, const CUtensorMap& w,
                   const CUtensorMap& out, const CUtensorMap& out_sh, const ExpertsParams& p,
                   int num_sms, cudaStream_t stream) {
  const size_t smem = 1024 + EX_BARS + 2 * EX_OUT + (size_t)EX_STAGES * EX_STAGE;
  auto kern = experts_pair_kernel<DOWN>;
  static bool configured_on[BF_MAX_DEVICES];
  bool& configured = configured_on[bf_current_device()];
  if (!configured) {
    cudaError_t ce =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (ce != cudaSuccess) return (int)ce;
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(EX_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(2 * (num_sms / 2), 1, 1);
  const cudaError_t ce = cudaLaunchKernelEx(&cfg, kern, a, a_sh, w, out, out_sh, p);
  if (ce != cudaSuccess) return (int)ce;
  return bf_launch_status();
}

}  // namespace

// x [T, width] (rows x_stride apart), w_gu [2 F, width], w_down [width, F] (rows ldd apart), all
// bfloat16; top_ids and top_w [T, top] and route_w [T, rw_cols] as the router leaves them.  max_tiles:
// T top / 256 + E; scratch: slot_of int [T top], row_w float [max_tiles 256], meta int [1 +
// max_tiles], xs bf16 [max_tiles 256, width], act bf16 [max_tiles 256, ff], act_sh bf16 [T, ff_sh],
// y float [max_tiles 256, width], y_sh float [T, width].
BF_EXPORT int bf_moe_grouped(const void* x, long long x_stride, const void* w_gu,
                             const void* w_down, long long ldd, const int* top_ids,
                             const float* top_w, const float* route_w, int rw_cols,
                             int shared_gate, int id_col, int T, int width, int E, int ff,
                             int ff_sh, int top, int max_tiles, int* slot_of, float* row_w,
                             int* meta, void* xs, void* act, void* act_sh, float* y, float* y_sh,
                             void* out, int act_kind, float limit, float shared_limit, float slope,
                             float up_offset, int num_sms, int* err, cudaStream_t stream) {
  if (T <= 0) return 0;
  const long long n = (long long)T * top;
  if (E < 1 || E > MG_MAX_EXPERTS || top < 1 || width % 8 || ff % 8 || ff_sh % 8 || ff <= 0 ||
      x_stride % 8 || ldd % 8 || num_sms < 2 || max_tiles < n / MG_TILE + E || n > (1 << 30) ||
      (act_kind != BF_ACT_SILU && act_kind != BF_ACT_CLAMPED) ||
      (((uintptr_t)x | (uintptr_t)w_gu | (uintptr_t)w_down | (uintptr_t)xs | (uintptr_t)act |
        (uintptr_t)act_sh | (uintptr_t)y | (uintptr_t)y_sh | (uintptr_t)out) & 15))
    return (int)cudaErrorInvalidValue;
  const int rows = max_tiles * MG_TILE, F = E * ff + ff_sh;
  CUtensorMap mxs, mx, mgu, mact, mact_st, msh, msh_st, mdown, my, mysh;
  int e;
  if ((e = bf_make_tensor_map_bf16_2d(&mxs, xs, rows, width, width, 128, BK)) ||
      (e = bf_make_tensor_map_bf16_2d(&mx, x, T, width, x_stride, 128, BK)) ||
      (e = bf_make_tensor_map_bf16_2d(&mgu, w_gu, 2LL * F, width, width, 64, BK)) ||
      (e = bf_make_tensor_map_2d_store(&mact_st, act, rows, ff, ff, 128, 2)) ||
      (e = bf_make_tensor_map_bf16_2d(&mact, act, rows, ff, ff, 128, BK)) ||
      (e = bf_make_tensor_map_bf16_2d(&mdown, w_down, width, F, ldd, 128, BK)) ||
      (e = bf_make_tensor_map_2d_store(&my, y, rows, width, width, 128, 4)))
    return e;
  msh = mact;
  msh_st = mact_st;
  mysh = my;
  if (ff_sh) {
    if ((e = bf_make_tensor_map_2d_store(&msh_st, act_sh, T, ff_sh, ff_sh, 128, 2)) ||
        (e = bf_make_tensor_map_bf16_2d(&msh, act_sh, T, ff_sh, ff_sh, 128, BK)) ||
        (e = bf_make_tensor_map_2d_store(&mysh, y_sh, T, width, width, 128, 4)))
      return e;
  }
  ExpertsParams p;
  p.tokens = T;
  p.width = width;
  p.E = E;
  p.ff = ff;
  p.ff_sh = ff_sh;
  p.F = F;
  p.rows = rows;
  p.meta = meta;
  p.row_w = row_w;
  p.sh_w = shared_gate ? route_w + E : nullptr;
  p.sh_w_stride = rw_cols;
  p.clamped = act_kind == BF_ACT_CLAMPED;
  p.gk = BfGateConst{limit, slope, up_offset};
  p.gk_sh = BfGateConst{shared_limit, slope, up_offset};
  p.err = err;
  moe_sort_kernel<<<1, 1024, 0, stream>>>(top_ids, top_w, (int)n, E, max_tiles, slot_of, row_w, meta);
  moe_gather_kernel<<<(unsigned)((n + 7) / 8), 256, 0, stream>>>(
      (const __nv_bfloat16*)x, x_stride, slot_of, (int)n, top, width, (__nv_bfloat16*)xs);
  if ((e = bf_launch_status())) return e;
  if ((e = experts_launch<false>(mxs, mx, mgu, mact_st, msh_st, p, num_sms, stream))) return e;
  if ((e = experts_launch<true>(mact, msh, mdown, my, mysh, p, num_sms, stream))) return e;
  const long long items = (long long)T * (width / 8);
  moe_combine_kernel<<<(unsigned)((items + 255) / 256), 256, 0, stream>>>(
      y, ff_sh ? y_sh : nullptr, slot_of, T, top, width, (const __nv_bfloat16*)x, x_stride, route_w,
      rw_cols, id_col, (__nv_bfloat16*)out);
  return bf_launch_status();
}
