// Keys and values of prompt portions in latent attention, expanded: the latents of a portion's whole
// context out of the pages into rows one behind the other, which one product then turns into every
// head's key and value (and prefill_attention_umma2 attends to).
//
// Attending in latent coordinates (attention_latent_mma.cu) needs no expansion but 576 + 512
// multiply-adds per score and head where expanded keys and values need 192 + 128; the expansion
// costs 256 x 512 per key and head, once for all of a portion's rows.  A prompt of a few hundred
// rows pays for it, a single token does not.  1,800 rows behind 500 cached keys, 16 heads: 964 us in
// latent coordinates (mma.sync, 91 TFLOP/s); 4.6 us for this kernel, 11 for the product and 60 for
// the attention (tcgen05; 432 TFLOP/s of the 26 GFLOP that are left), and the two products that
// carry queries into latent coordinates and results out of them fall away (for the single tokens of a
// mixed step they stay: for their rows alone where they come first, as the scheduler puts them, else
// for all rows).  The layer: 1,061 -> 143 us.
#include "common.cuh"

// A warp per row.  Portion i's keys (items[i]: request, first token row, rows, first position) take
// the rows from the sum of the earlier portions' contexts, each rounded up to 64, on; the rows
// between its last key and the next multiple of 64 become zero.  kv_base[i]: that first row.
__global__ void latent_gather_kernel(const __nv_bfloat16* __restrict__ cache,
                                     const int* __restrict__ tables, int table_stride,
                                     const int* __restrict__ items, int n_items,
                                     __nv_bfloat16* __restrict__ lat,
                                     __nv_bfloat16* __restrict__ rot, int* __restrict__ kv_base,
                                     int rows, int rank, int dr, int page_size, int num_pages,
                                     int* __restrict__ err) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= rows) return;
  int base = 0, seq = -1, key = 0, ctx = 0;
  for (int i = 0; i < n_items; ++i) {
    const int* it = items + 4 * i;
    const int n = it[3] + it[2];
    if (row == 0 && lane == 0) kv_base[i] = base;
    const int next = base + (n + 63) / 64 * 64;
    if (row >= base && row < next) {
      seq = it[0];
      key = row - base;
      ctx = n;
      if (row > 0) break;
    }
    base = next;
  }
  bool ok = seq >= 0 && key < ctx;
  const __nv_bfloat16* src = cache;
  if (ok) {
    const int lp = key / page_size;
    const int page = tables[(size_t)seq * table_stride + lp];
    if (page < 0 || page >= num_pages) {
      if (lane == 0) atomicOr(err, BF_ERR_PAGE);
      ok = false;
    } else {
      src = cache + ((size_t)page * page_size + (key - lp * page_size)) * (rank + dr);
    }
  }
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint4* s4 = reinterpret_cast<const uint4*>(src);
  uint4* l4 = reinterpret_cast<uint4*>(lat + (size_t)row * rank);
  uint4* r4 = reinterpret_cast<uint4*>(rot + (size_t)row * dr);
  for (int c = lane; c < rank / 8; c += 32) l4[c] = ok ? s4[c] : zero;
  for (int c = lane; c < dr / 8; c += 32) r4[c] = ok ? s4[rank / 8 + c] : zero;
}

BF_EXPORT int bf_latent_gather(const void* cache, const int* tables, int table_stride,
                               const int* items, int n_items, void* lat, void* rot, int* kv_base,
                               int rows, int rank, int dr, int page_size, int num_pages, int* err,
                               cudaStream_t stream) {
  if (rows <= 0 || n_items <= 0) return 0;
  if (rank % 8 || dr % 8 || ((uintptr_t)cache & 15) || ((uintptr_t)lat & 15) ||
      ((uintptr_t)rot & 15))
    return (int)cudaErrorInvalidValue;
  latent_gather_kernel<<<(rows + 7) / 8, 256, 0, stream>>>(
      (const __nv_bfloat16*)cache, tables, table_stride, items, n_items, (__nv_bfloat16*)lat,
      (__nv_bfloat16*)rot, kv_base, rows, rank, dr, page_size, num_pages, err);
  return bf_launch_status();
}
