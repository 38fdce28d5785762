// Where the key-block kernels of the backward leave dS for the GEMMs of bwd_ds_gemm_sm100.cu.
//
// dS of one head is cut into tiles of 128 queries x 128 keys, 16-bit, 32 KB each; only tiles that the mask leaves exist, row of
// tiles by row of tiles. Inside a tile: [16 groups of 8 queries][128 keys][8 queries]. A thread that owns a key writes 16 bytes
// next to its neighbours' (512 contiguous bytes per warp and store), and the same bytes are an operand of tcgen05.mma without
// swizzle in both directions: keys as the contraction (dQ = dS K, MN-major A) and queries as the contraction (dK = dS^T Q, K-major).
#pragma once

#include <stdint.h>

namespace sdpa_b200 {

constexpr int kDsTile = 128;
constexpr size_t kDsTileBytes = static_cast<size_t>(kDsTile) * kDsTile * 2;

struct DsTiles {
  uint16_t* data;           // null: nobody wants dS
  const int32_t* seq_base;  // packed: tiles of one head in front of each sequence; null: dense
  int head0;                // dense: batch * heads_q index of the first head in the buffer
  uint32_t capacity;        // tiles in the buffer
};

// Key tiles that query tile `qt` sees under a bottom-right causal mask are [0, clamp(qt + shift, 0, key_tiles)).
__host__ __device__ inline int ds_shift(int len_q, int len_k, bool causal) {
  return causal ? (len_k - len_q + 2 * kDsTile - 1) >> 7 : (len_k + kDsTile - 1) / kDsTile;
}

// Tiles in front of row of tiles `qt`: the sum of clamp(i + shift, 0, key_tiles) over i < qt.
__host__ __device__ inline int64_t ds_row_start(int qt, int key_tiles, int shift) {
  const int lo = shift < 0 ? (-shift < qt ? -shift : qt) : 0;      // rows that see nothing
  int full = key_tiles - shift;                                    // from here on a row sees every key
  full = full < lo ? lo : (full > qt ? qt : full);
  return static_cast<int64_t>(full - lo) * (lo + full - 1 + 2 * static_cast<int64_t>(shift)) / 2 +
         static_cast<int64_t>(qt - full) * key_tiles;
}

__host__ __device__ inline int64_t ds_tiles_per_head(int len_q, int len_k, bool causal) {
  if (len_q <= 0 || len_k <= 0) return 0;
  return ds_row_start((len_q + kDsTile - 1) / kDsTile, (len_k + kDsTile - 1) / kDsTile, ds_shift(len_q, len_k, causal));
}

// The tiles of one head of one (sequence's) problem.
struct DsHead {
  int64_t base;
  int key_tiles, shift;
  __device__ __forceinline__ uint32_t tile(int qt, int kt) const {
    return static_cast<uint32_t>(base + ds_row_start(qt, key_tiles, shift) + kt);
  }
};

__device__ __forceinline__ DsHead ds_head(const DsTiles& ds, int b, int head_q, int heads_q, int len_q, int len_k, bool causal) {
  DsHead h;
  h.key_tiles = (len_k + kDsTile - 1) / kDsTile;
  h.shift = ds_shift(len_q, len_k, causal);
  const int64_t per_head = ds_tiles_per_head(len_q, len_k, causal);
  h.base = ds.seq_base != nullptr ? static_cast<int64_t>(ds.seq_base[b]) * heads_q + head_q * per_head
                                  : (static_cast<int64_t>(b) * heads_q + head_q - ds.head0) * per_head;
  return h;
}

// Eight queries (one 16-byte group) of one key.
__device__ __forceinline__ uint4* ds_group(const DsTiles& ds, uint32_t tile, int query_group, int key) {
  return reinterpret_cast<uint4*>(ds.data) + static_cast<size_t>(tile) * (kDsTileBytes / 16) + query_group * kDsTile + key;
}

// Entry b of DsTiles::seq_base, by one block of a pre-pass: the tiles of one head of the sequences in front of sequence b.
__device__ __forceinline__ void write_seq_base(int32_t* seq_base, const int32_t* cu_q, const int32_t* cu_k, int b, bool causal) {
  __shared__ int tiles_before;
  if (threadIdx.x == 0) tiles_before = 0;
  __syncthreads();
  int mine = 0;
  for (int i = threadIdx.x; i < b; i += blockDim.x)
    mine += static_cast<int>(ds_tiles_per_head(cu_q[i + 1] - cu_q[i], cu_k[i + 1] - cu_k[i], causal));
  if (mine != 0) atomicAdd(&tiles_before, mine);
  __syncthreads();
  if (threadIdx.x == 0) seq_base[b] = tiles_before;
}

}  // namespace sdpa_b200
