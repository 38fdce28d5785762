// The GEMMs of the backward that read dS from the workspace (bwd_ds_gemm_sm100.cu).
#pragma once

#include "ds_tiles.cuh"
#include "kernels.h"

namespace sdpa_b200 {

// How a call's dS goes through the workspace: `kv_heads` (batch * heads_kv indexes) per pass, `tiles` of room, none if 0.
struct DsPlan {
  int kv_heads = 0;
  uint32_t tiles = 0;
};

DsPlan ds_plan(const sdpa_b200_params& p);
size_t ds_table_bytes(const sdpa_b200_params& p);  // DsTiles::seq_base, in front of the tiles
size_t ds_workspace_bytes(const sdpa_b200_params& p, const DsPlan& plan);

struct DsGemmParams {
  DsTiles ds;
  const int32_t* cu_q;
  const int32_t* cu_k;
  uint32_t* counter;  // next unit; cleared by the kernel in front
  uint32_t* status;
  uint16_t* dq;       // bf16 or f16 bits
  uint16_t* dk;
  int64_t dq_row_stride, dq_head_stride, dk_row_stride, dk_head_stride;
  int seqlen_q, seqlen_k, heads_q, heads_kv, kv_group, head_dim;
  int is_causal;
  float scale;
  // units: groups of `heads_per_group` KV heads; in a group the 256-row key units (dK), then the 256-row query units (dQ)
  int kv_head0, num_kv_heads;  // batch * heads_kv indexes this launch covers
  int num_groups, heads_per_group, key_units_per_group, units_per_group, query_pairs, key_pairs;
  uint32_t units;
};

// dQ of the query heads of KV heads [kv_head0, kv_head0 + num_kv_heads) (batch * heads_kv indexes), and their dK `with_dk`. The
// kernel in front in the stream has written their dS tiles, cleared `counter` and may signal launch_dependents early.
int launch_bwd_ds_gemm(const sdpa_b200_params& p, const DsTiles& ds, int kv_head0, int num_kv_heads, bool with_dk,
                       uint32_t* counter, uint32_t* status, cudaStream_t stream);

// 2-D map over the dS tiles as rows of 256 8-byte words (one group of 8 queries x 128 keys each), no swizzle.
int make_ds_tensor_map(CUtensorMap* map, const void* base, uint32_t tiles, int box_words, int box_rows);

}  // namespace sdpa_b200
