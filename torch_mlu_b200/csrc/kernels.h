// Internal launch interface between the C-ABI front end (sdpa_api.cu) and the kernel files.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/sdpa_b200.h"

namespace sdpa_b200 {

// First 256 bytes of every workspace: word 0 is the device status, the rest is reserved.
constexpr size_t kWorkspaceHeaderBytes = 256;

// Thread-local error text (set by whoever returns a non-OK status).
void set_error(const char* fmt, ...);
void count_launch(int n = 1);

// Builds a 4-D tensor map over 16-bit elements (f16 or bf16) {head_dim, rows, heads, batch} with a
// {64, box_rows, 1, 1} box and 128-byte swizzle. Strides are in ELEMENTS. Returns an SDPA_B200_* status.
int make_tensor_map_16(bool f16, CUtensorMap* map, const void* base, int head_dim, int64_t rows,
                       int64_t heads, int64_t batch, int64_t row_stride, int64_t head_stride,
                       int64_t batch_stride, int box_rows);

// Prefill forward (TMA + tcgen05), a persistent kernel with one CTA per SM.
int launch_fwd_prefill(const sdpa_b200_params& p, void* workspace, cudaStream_t stream);

// Forward for head dims above 128 (up to 256): one CTA per 128 query rows, Q in tensor memory (d256_sm100.cu).
int launch_fwd_d256(const sdpa_b200_params& p, void* workspace, cudaStream_t stream);
// Backward for the same head dims: a pre-pass, a kernel for dV and dS and the GEMMs for dK and dQ, or, without room for dS, one
// kernel each for dV, dK and dQ (d256_sm100.cu).
size_t bwd_d256_workspace_min_bytes(const sdpa_b200_params& p);
size_t bwd_d256_workspace_bytes(const sdpa_b200_params& p);
int launch_bwd_d256(const sdpa_b200_params& p, void* workspace, size_t workspace_bytes, cudaStream_t stream);

// Kernels take (batch, head) pairs in groups whose streamed tensors stay in L2 together, and the blocks of a group heaviest first.
// Heads per group, from the bytes that one head streams (packed: at the longest length). The groups are of one size, as far as that goes: a small
// last group puts its few heavy blocks where no light ones are left to fill up behind them (us, filled up | even: forward D256, B3 H12, 1479 rows of
// 2047, 15 + 15 + 6 heads or 3 x 12 95.3 | 89.2, 12 packed sequences of 300 to 2000, 16/4 332 | 312, D128, 16 of 512 to 4096, 32/8 915 | 885; step of
// B3 H12 L1479 D128 143 | 133, of B5 H8 L2500 D192 551 | 544). Not (`even`) in the fused kernel (step of B5 H12 L1500 D64 154.6 | 156.4), nor in packed backwards
// without a mask, whose heads stand by sequence: even groups cut the sequences elsewhere, and where the last group begins inside the longest one it has
// the longest chains (722, 529, 2016 and 843 tokens, 32/8 heads, D128, 12 + 12 + 8 or 11 + 11 + 10 heads: dK/dV 197 | 252 us).
inline int heads_per_l2_group(double bytes_per_head, int num_heads, double group_bytes = 48.0 * 1024 * 1024, bool even = true) {
  int n = static_cast<int>(group_bytes / bytes_per_head);
  n = n > 32 ? 32 : (n < 1 ? 1 : n);
  if (n >= num_heads) return num_heads;
  const int groups = (num_heads + n - 1) / n;
  return even ? (num_heads + groups - 1) / groups : n;
}

// Forward: smaller groups, so that more CTAs read the same K and V at a time (B4 H32 L4096 D128 causal 539 us with groups of 48 MB, 531 of 32,
// 527 of 16; unmasked, 16 heads 503, 497, 491; B2 H32 L8192 causal 1022, 998, 996; but B2 H16 L3000 causal 89.1, 88.6, 91.7;
// head_dim 256, B4 H16 L4096 causal 544, 534).
constexpr double kForwardGroupBytes = 32.0 * 1024 * 1024;

// Forward under a causal mask, up to head_dim 128: how many of the lightest ranks of blocks come behind all groups, over all heads. With whole
// groups to the end the CTAs that had taken the last group's heavy blocks ran on alone: the longest-running CTA against the mean 280 to 233
// thousand cycles at B8 H16 L2048 D128, 911 to 825 at B4 H32 L4096; now 240 to 231 and 821 to 806. Calls over seconds, with the late claims of
// the forward: these two 172 us -> 166 and 568 -> 533, B2 H16 L3000 101 -> 88.6, B4 H32/8 L1000 57.7 -> 51.4, 9 packed sequences of 29 to 2820
// tokens, 8/1, D64 92.8 -> 72.8. As many as half, and as stay in L2 together, since heads do not share K and V at a time there: `bytes_per_rank`
// are those that one more rank makes all heads stream, `prefix_bytes` those that every rank does, since the keys in front of the first query are
// visible to all (limit of 128 MB: 555 us at L4096, 64: 539, 32: 538; B8 H16 L2048 170, 169, 166. With the prefix left out of the count, 512 rows behind a
// cached prefix read all of K and V twice, us, so | counted: B7 H32 512 of 1297 102.5 | 92.6, B8 H32 512 of 2048 156.8 | 147.1, B4 H32 1024 of 4096
// 282 | 259, B8 H32 1152 of 1984 D96 267 | 259). Not
// where the hardware deals out CTAs of single blocks: it claims as late as can be, and the kernel ends within 2 % of the mean CTA as it is
// (head_dim 256 forward, B4 H16 L4096 534 without, 533 with; B8 H16 L644 80, 82; backward, step of B4 H16 L1024 D256 227, 231, of B8 H12 L1000
// D64 135, 159).
inline int tail_ranks(int ranks, double bytes_per_rank, double prefix_bytes) {
  const double fit = (32.0 * 1024 * 1024 - prefix_bytes) / bytes_per_rank;
  return fit < 1 ? 0 : fit < ranks / 2 ? static_cast<int>(fit) : ranks / 2;
}

// Packed backward under a causal mask, from what all sequences together stream: the longest one says little about it, and in fewer and
// larger groups fewer long chains start late. Groups stream 112 MB, except in the fused kernel, which also adds into its accumulator (20
// sequences of 100 to 3000 tokens, D64: step 1048 us by the longest, 1074 so) (dK/dV kernel of 12 sequences of 64 to 2048 tokens, 16/4
// heads: 153 us in five groups, the last 50 of them with idle SMs, 134 in one; step 365 -> 350, with 64 MB 360). Without a mask all blocks
// of a sequence are equally heavy, and the order by block index in groups by the longest sequence is the faster one (step of 20
// sequences of 300 to 3000 tokens, 16/4 heads, D128: 2909 us, by all bytes and by the blocks behind 3066; 6 of 50 to 4000, 32/8: 2905,
// 2983; 12 of 500 to 1000, 16/16: 451, 468). The dS GEMM, which takes its units from a counter, always goes by all bytes.
inline int heads_per_packed_group(double all_bytes, int num_heads) {
  const int groups = 1 + static_cast<int>(all_bytes / (112.0 * 1024 * 1024));
  return (num_heads + groups - 1) / groups;
}

// Launches `kernel` in clusters of `cluster` CTAs; with `overlap` so that its CTAs may start as soon as every CTA of the grid in front of it in the stream has said that it may
// (launch_dependents) or has left, and an SM has room: its launch and set-up then pass under that grid's tail. The kernel waits
// (wait_for_previous_grid) before it touches global memory. Not under stream capture, where what stands in front may be no kernel.
template <typename... Params, typename... Args>
cudaError_t launch_behind(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, bool overlap, int cluster, const Args&... args) {
  if (overlap) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    overlap = cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    if (!overlap) (void)cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (overlap) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, args...);
  return err == cudaSuccess ? cudaGetLastError() : err;
}

// Forwards that are launched behind the kernel in front of them: up to 1e11 operations. Longer ones have little to hide and run into the power
// cap, where the gap costs nothing and filling it does. (Calls back to back, early | plain start, us: 1.3e11 operations, D128, B2 H32/8, 512 rows of 8192
// 126 | 122, B1 H32/8, 1024 of 8192 122 | 120; 6e10, B2 H32/8, 512 of 4096 66.9 | 67.0; but 8e10, B1 H9 L4096 unmasked 66.5 | 68.1; 7e10, D256, B3 H12,
// 1479 of 2047 95.3 | 97.5; 3e10, D128, B1 H32/8, 512 of 4096 55.3 | 56.1.)
inline bool short_forward(const sdpa_b200_params& p) {
  const double rows = p.cu_seqlens_q != nullptr ? p.total_q : static_cast<double>(p.batch) * p.max_seqlen_q;
  const double hidden = p.is_causal ? (p.max_seqlen_q < p.max_seqlen_k ? p.max_seqlen_q : p.max_seqlen_k) / 2.0 : 0.0;
  return 4.0 * p.head_dim * p.heads_q * rows * (p.max_seqlen_k - hidden) <= 1e11;
}

// Number of SMs of the current device (cached per device), <= 0 on error.
int sm_count();

// Split-KV decode forward. Workspace layout is private to decode_splitkv.cu.
size_t decode_workspace_bytes(const sdpa_b200_params& p);
int launch_fwd_decode(const sdpa_b200_params& p, void* workspace, size_t workspace_bytes,
                      cudaStream_t stream);

// Argument checks of the forward entry point (no device is touched) and the device check, for entry
// points defined outside sdpa_api.cu. Each returns an SDPA_B200_* status and sets the error text.
int validate_forward_args(const sdpa_b200_params* p);
int check_device();

// Refuses what the split-KV decode kernels have no code for (packed tensors, seqlen_q != 1, head dims other
// than 64 and 128, dropout, bias). Touches no device.
int check_decode_request(const sdpa_b200_params& p);

// round(dropout_p * 256), the byte threshold of the dropout keep-masks (dropout_mask.cu)
uint32_t dropout_drop_byte(float dropout_p);

// Backward up to head_dim 128: delta pre-pass, then the kernels that bwd_sm100.cu chooses. A call that is given at least the least
// workspace runs; with less than bwd_workspace_bytes() on other kernels.
size_t bwd_workspace_min_bytes(const sdpa_b200_params& p);
size_t bwd_workspace_bytes(const sdpa_b200_params& p);
int launch_bwd(const sdpa_b200_params& p, void* workspace, size_t workspace_bytes,
               cudaStream_t stream);

}  // namespace sdpa_b200
