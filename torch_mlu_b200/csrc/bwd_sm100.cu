// Backward attention kernels for sm_100a.
//
// Replaces the device work behind mha_varlen_bwd -> cnnlFlashAttentionBackward
// (torch_mlu/csrc/aten/operators/cnnl/internal/FlashAttention_internal.cpp:449-480):
// given dO, Q, K, V, O and the saved logsumexp, recompute P = exp(scale*QK^T - lse) and
//   dV = P^T dO,  dP = dO V^T,  dS = P o (dP - delta),  dQ = scale dS K,  dK = scale dS^T Q
// with delta = rowsum(dO o O). GQA: dK/dV of one KV head sum over its query heads inside one
// CTA, so nothing is accumulated with atomics and results are bit-reproducible. With dropout (kDrop
// instances) dV takes P o M / (1 - p) and dS = P o (M o dP / (1 - p) - delta); with an additive bias (kBias
// instances) the scores are scale*QK^T + bias and the dQ kernel also writes dS as the bias gradient.
//
// Three launches, of which the last two are one where the same instance serves both (bwd_tile_kernel_pair):
//   1. bwd_preprocess_kernel: delta and the log2-domain logsumexp into a padded
//      [batch, heads_q, ceil128(max_seqlen_q)] workspace (rows past a sequence get lse = +inf,
//      which later turns their P into exact zeros).
//   2. bwd_tile_kernel<kModeDKDV>: one CTA, or a cluster that shares the query heads (bwd_split), per (batch, kv head,
//      128-key block). K and V tiles
//      stay in shared memory; (Q, dO) tiles (of 128 rows, up to head_dim 64 of 64 unless wide_tiles()) stream through a TMA ring. Per Q tile:
//      S^T = K Q^T and dP^T = V dO^T on tcgen05 into TMEM, two compute warpgroups (thread = key
//      row = TMEM lane, one warpgroup per half of the tile's queries) form P^T and dS^T, write
//      them back to TMEM as bf16, and MMAs with the TMEM operand accumulate dV += P^T dO and
//      dK += dS^T Q (the streamed tiles are re-read in place as MN-major operands).
//   3. dQ, one of: bwd_tile_kernel<kModeDQ>, one CTA per (batch, query head, 128-query block); Q and dO
//      stay, (K, V) stream; S = Q K^T, dP = dO V^T, dS -> TMEM, dQ += dS K. Or, where launch 2 has left its dS
//      in the workspace as well (8 stores of 16 bytes per thread and item: 281 -> 308 us at B8 H16 L2048 D128
//      causal), the GEMM of bwd_ds_gemm_sm100.cu, which forms no scores (221 us -> 122).
// TMEM: T1 [0,128) T2 [128,256) ACC1 [256,384) ACC2 [384,512); up to head_dim 64 accumulators of 64 columns, with tiles of 64 rows four times 64. The bf16 P and dS of an item both
// live in the item's score buffer, so the buffer that held dP is free as soon as it has been read;
// the MMA issuer uses that (and, for dQ, the unused ACC2) to run the next item's score GEMMs and
// exponentials under the current item's accumulation MMAs (buffer schedule at the issuer).
#ifdef SDPA_BWD_STAMPS
#include <cstdlib>
#endif

#include <algorithm>
#include <type_traits>
#include <utility>

#include "bwd_common.cuh"
#include "bwd_ds_gemm.h"
#include "packed_grads.cuh"

namespace sdpa_b200 {
namespace {

// Streamed tiles (kY rows). Up to head_dim 64 they have 64 rows where launches fill the GPU, so that a CTA's score buffers and accumulators take half of the tensor memory and
// two CTAs share an SM: the one's exponentials run under the other's MMAs and waits, set-ups and epilogues. Above, the accumulators leave
// no room for that. One chain of 128-row items per SM took as long as at head_dim 128. (Step of B8 H12 L512 with a mask 94.3 -> 88.9 us, B16
// 153 -> 134, B8 H16 L2048 579 -> 526, B4 H12 L600 with a learned bias 152 -> 144. One warpgroup with 64 columns instead: 97.) Where CTAs are few, a chain of 128-row items has
// half as many and is over sooner: wide_tiles().
constexpr int kComputeWarps = 8;  // two warpgroups, each with half of an item's columns
template <int kY>
constexpr int kThreads = (kComputeWarps + (kY == 64 ? 4 : 3)) * 32;  // compute, TMA producer, two MMA issuers (and an idle warp)
// Register hand-over of the instances with two CTAs per SM (setmaxnreg; launched with 80). What the third warpgroup releases
// covers what the other two take, or the increase would wait forever.
constexpr int kRegsCompute = 96, kRegsOther = 48;
static_assert(2 * kRegsCompute + kRegsOther <= 3 * 80, "setmaxnreg.inc would wait forever");

// Ring of streamed tiles Y1(0), Y2(0), Y1(1), Y2(1), ...: 4 slots of 32 KB (8 of 8 KB) for dK/dV, which also stages
// the per-query vectors, 5 for dQ so that K(i+2) can land while item i is still accumulating.
constexpr int kMaxStages = 8;
__host__ __device__ constexpr int stages_for(int mode, int d) { return mode == 1 ? 5 : d == 64 ? 8 : 4; }
constexpr int kModeDKDV = 0;
constexpr int kModeDQ = 1;

__host__ __device__ constexpr uint32_t x_bytes(int d) { return kTile * d * 2; }                     // one stationary tile
__host__ __device__ constexpr uint32_t y_bytes(int d, int y) { return y * d * 2; }            // one streamed tile
constexpr uint32_t kSmemX = 0;                                   // stationary pair
__host__ __device__ constexpr uint32_t smem_y_off(int d) { return 2 * x_bytes(d); }
__host__ __device__ constexpr uint32_t smem_vec_off(int mode, int d, int y) { return smem_y_off(d) + stages_for(mode, d) * y_bytes(d, y); }
// per-slot (lse2[128], delta[128]), dK/dV only
__host__ __device__ constexpr uint32_t smem_bar_off(int mode, int d, int y) { return smem_vec_off(mode, d, y) + (mode == 1 ? 0 : stages_for(mode, d) * 1024); }
// behind the barriers, dQ with a key bias only: 64 16-bit bias values per compute warp
__host__ __device__ constexpr uint32_t smem_key_bias_off(int mode, int d, int y) { return smem_bar_off(mode, d, y) + 256; }
// at least 80 KB: a third CTA on the SM would wait for tensor memory
__host__ __device__ constexpr uint32_t smem_bytes_for(int mode, int d, int y, bool key_bias) {
  const uint32_t used = smem_key_bias_off(mode, d, y) + (mode == 1 && key_bias ? 8 * 128 : 0) + 1024;
  return used > 80 * 1024 ? used : 80 * 1024;
}
constexpr uint32_t kBarXFull = 0;
constexpr uint32_t kBarYFull = 8;
constexpr uint32_t kBarYEmpty = kBarYFull + 8 * kMaxStages;
constexpr uint32_t kBarSFull = kBarYEmpty + 8 * kMaxStages;   // 2: first score GEMM (X1 Y1^T) of an item done
constexpr uint32_t kBarDFull = kBarSFull + 16;             // second score GEMM (X2 Y2^T) done
constexpr uint32_t kBarDFree = kBarDFull + 8;              // all compute warps have read dP out of TMEM
// Of the next two there is one per item parity: in the dQ kernel the compute warps can complete the next item's P / dS, in the dK/dV kernel its
// P, before the accumulation issuer has looked at this one's, and to a wait on a parity two phases further on read "not yet". The item
// after that needs the issuer first.
constexpr uint32_t kBarPFull = kBarDFree + 16;             // 2: all compute warps have stored P / dS
constexpr uint32_t kBarAccFull = kBarPFull + 16;
constexpr uint32_t kBarP1Full = kBarAccFull + 8;           // 2, dK/dV: all compute warps have stored P (dS still to come)
constexpr uint32_t kBarWFree = kBarP1Full + 16;            // 2 (item parity): the accumulation GEMMs have read P / dS
constexpr uint32_t kBarSIssued = kBarWFree + 16;           // dK/dV: the next item's score GEMM is in the pipe
constexpr uint32_t kBarEpiFull = kBarSIssued + 8;           // all compute warps have staged their output rows
constexpr uint32_t kSmemTmemPtr = kBarEpiFull + 8;
constexpr uint32_t kSmemAbort = kSmemTmemPtr + 4;
static_assert(kSmemAbort + 4 <= 256, "the barriers reach into the key bias");

// Profiling builds (-DSDPA_BWD_STAMPS) time-stamp pipeline events of one CTA per kernel; role 0/1 =
// lane 0 of the first warp of each compute warpgroup, roles 2 and 3 = the MMA issuer.
#ifdef SDPA_BWD_STAMPS
#define BWD_STAMP(role, item, ev)                                                                       \
  do {                                                                                                  \
    if (stamp_on && (item) < 24)                                                                        \
      p.stamps[((kMode * 4 + (role)) * 24 + (item)) * 8 + (ev)] = static_cast<float>(clock64() - t_start); \
  } while (0)
#else
#define BWD_STAMP(role, item, ev) do {} while (0)
#endif

// What a tile kernel instance does about an additive bias. kKeyBias: one that is the same for every query (a key-padding mask,
// ALiBi-like slopes) and whose gradient nobody wants. It joins the per-row addend of the exponent: one value per thread in the
// dK/dV kernel; in the dQ kernel 64 values per warp and item, fetched as one word per lane under the waits and read back
// as broadcasts. The general loads keep 32 more registers alive per thread. Backward of B8 H12 L512 D64 with a padding mask, all
// launches: 61.5 us; in the fused kernel, whose dQ varies in its last bits from call to call, 60.3.
enum BiasKind { kNoBias = 0, kFullBias = 1, kKeyBias = 2 };

// kDsCall: the call's dS goes through the workspace where there is room (launch_bwd). An instance of its own, since with both kinds of
// exponentials and the dS stores behind branches the calls without dS were slower (dK/dV and dQ kernel of 6 packed sequences of 50 to 4000
// tokens, 32/8 heads, unmasked: 1222 + 1076 us, so 1137 + 1019).
// kPair: the CTA is one of a grid that does both, with `block` its index among those of its kind.
template <int kMode, int kD, bool kF16, bool kDrop, int kBias, bool kDsCall, bool kSplit, int kY, bool kPair>
__device__ __forceinline__ void tile_cta(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_do,
                                         const CUtensorMap& tm_o1, const CUtensorMap& tm_o2, const BwdKernelParams& p, const BlockOrder& order,
                                         int heads_x, int block) {
  extern __shared__ uint8_t smem_raw[];
#ifdef SDPA_BWD_STAMPS
  const long long t_entry = clock64();
#endif
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // dK/dV: the pre-pass in front signals at once that this grid may start, so its set-up and the first K and V loads run under the
  // pre-pass's tail; its vectors are read behind the wait for it. The kernel behind (the dQ kernel, which depends on nothing
  // written here, or the dQ GEMM, which waits for this grid) is let in by every CTA behind that wait, so that it too finds the
  // vectors complete. CTAs without work wait as well: a grid must not complete before the one in front of it.
  if (kMode == kModeDKDV && kDsCall && p.ds.data != nullptr && block == 0 && threadIdx.x == 0)
    *p.ds_counter = 0u;  // read by the dQ GEMM behind its wait for this grid; here, since block 0 may be one without work
  constexpr int kStages = stages_for(kMode, kD);
  constexpr int kC = kY / 2;  // columns per compute warpgroup, i.e. per thread
  constexpr int kTmaWarp = kComputeWarps, kScoreWarp = kTmaWarp + 1, kAccWarp = kTmaWarp + 2;
  constexpr uint32_t kTmemCols = kY == 64 ? 256 : 512;
  static_assert(2 * kY + 2 * kD <= static_cast<int>(kTmemCols), "score buffers and accumulators");
  constexpr uint32_t kXBytes = x_bytes(kD), kYBytes = y_bytes(kD, kY);
  constexpr uint32_t kSmemY = smem_y_off(kD);
  constexpr uint32_t kSmemVec = smem_vec_off(kMode, kD, kY);
  constexpr uint32_t kSmemBar = smem_bar_off(kMode, kD, kY);
  constexpr int kBoxRows = kD == 64 ? 64 : kTile;  // of the maps that load; a tile of 128 rows takes two boxes of 64
  constexpr uint32_t kBoxBytes = kBoxRows * kD * 2;

  // CTA order (1-D grid, block_order.cuh): heaviest blocks first (dK/dV: key block 0 sees every query; dQ: the last query block sees
  // every key). Packed, causal: blocks with the same number of blocks behind (dQ: in front of) them in their own
  // sequence count as equally heavy, so that a short sequence's first key block does not go before a long one's second.
  int b, hx, xb;
  {
    int rank, bh;
    if (!block_of_slot(order, kSplit ? block / p.split : block, rank, bh)) {
      wait_for_previous_grid();
      return;
    }
    bh += p.bh0;
    xb = (kMode == kModeDKDV) ? rank : order.ranks - 1 - rank;
    b = bh / heads_x;
    hx = bh - b * heads_x;
  }
  int q_off = 0, k_off = 0, len_q = p.seqlen_q, len_k = p.seqlen_k, bcoord = b;
  if (p.cu_q != nullptr) {
    q_off = p.cu_q[b];
    len_q = p.cu_q[b + 1] - q_off;
    k_off = p.cu_k[b];
    len_k = p.cu_k[b + 1] - k_off;
    bcoord = 0;
    if (kMode == kModeDKDV && p.is_causal) xb -= order.ranks - (len_k + kTile - 1) / kTile;
  }
  const int causal_off = len_k - len_q;
  const int len_x = (kMode == kModeDKDV) ? len_k : len_q;
  const int x0 = xb * kTile;
  if (x0 < 0 || x0 >= len_x) {
    wait_for_previous_grid();
    return;
  }

  // streamed tile range [y_lo, y_hi) (in tiles of kY rows) per head, and heads per CTA
  int y_lo = 0, y_hi = 0;
  if (kMode == kModeDKDV) {
    y_hi = (len_q + kY - 1) / kY;
    if (p.is_causal) y_lo = max(0, (x0 - causal_off) / kY);  // first query tile with a row >= x0 - off
    if (p.is_causal && x0 - causal_off > len_q - 1) y_lo = y_hi;
  } else {
    int vis_end = len_k;
    if (p.is_causal) vis_end = min(len_k, x0 + kTile + causal_off);
    y_hi = vis_end > 0 ? (vis_end + kY - 1) / kY : 0;
  }
  const int tiles_per_head = max(0, y_hi - y_lo);
  // dK/dV: the CTAs of a cluster (kSplit) take equal shares of the group's query heads
  const int cluster_rank = kSplit ? block % p.split : 0;
  const int heads_here = kSplit ? p.kv_group / p.split : (kMode == kModeDKDV) ? p.kv_group : 1;
  const auto query_head = [&](int hi) { return hx * p.kv_group + (kSplit ? cluster_rank * heads_here : 0) + hi; };
  const int n_items = tiles_per_head * heads_here;

  const uint32_t bar = base + kSmemBar;
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + kSmemBar + kSmemAbort);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(smem + kSmemBar + kSmemTmemPtr);

  // TMA producer state. The producer thread also initialises the barriers and issues the first loads
  // (the stationary pair and the first kPreloaded ring tiles, whose slots are free by construction)
  // BEFORE the set-up barrier, so that their latency runs under the TMEM allocation.
  const CUtensorMap* tmx1 = (kMode == kModeDKDV) ? &tm_k : &tm_q;
  const CUtensorMap* tmx2 = (kMode == kModeDKDV) ? &tm_v : &tm_do;
  const CUtensorMap* tmy1 = (kMode == kModeDKDV) ? &tm_q : &tm_k;
  const CUtensorMap* tmy2 = (kMode == kModeDKDV) ? &tm_do : &tm_v;
  const int x_row = ((kMode == kModeDKDV) ? k_off : q_off) + x0;
  const int y_off = (kMode == kModeDKDV) ? q_off : k_off;
  constexpr int kPreloaded = kMode == kModeDQ ? 4 : kStages;
  // ring tile idx: Y1(idx/2) if even, Y2(idx/2) if odd; false when a wait gave up
  auto load_tile = [&](int idx) -> bool {
        const int i = idx >> 1;
        int s = idx % kStages;
        uint32_t use = static_cast<uint32_t>(idx / kStages);
        if (kMode == kModeDQ) {  // K ring: slots 0-2, V ring: slots 3-4
          s = (idx & 1) ? 3 + (i & 1) : i % 3;
          use = static_cast<uint32_t>((idx & 1) ? (i >> 1) : i / 3);
        }
        // Slot reuse. dK/dV: the pair of slots of item i - 2 is released by one commit behind its
        // accumulation GEMMs. dQ has no release commits (they cost the issuer time) and watches a
        // barrier the GEMMs signal anyway: the score-full barrier of S(i-1), waited for before K(i).
        //   K(i) reuses the slot of K(i-3), last read by dQ(i-3); V(i) reuses the slot of V(i-2), read
        //   by dP(i-2) only. S(i-1) overwrites the buffer of dS(i-3), so its issuer has waited for
        //   dQ(i-3) (`W free`), and it issues dP(i-2) before S(i-1) itself (prologue: S0 dP0 S1; item j:
        //   dP(j+1), S(j+2)); the tensor pipe keeps the order of one thread's MMAs. So "S(i-1) done"
        //   covers both slots; V(i) is loaded right behind K(i) and needs no wait of its own.
        //   A parity wait can only tell "this phase is over" from "it is not" while the barrier is at
        //   most one phase further on. That holds here: the next phase of this barrier is S(i+1), and
        //   S(i+1) needs K(i+1), which this loop loads later. (The dP-full barrier would NOT do for
        //   V(i): dP(i-1) can finish as well before the producer looks, and two phases on the parity
        //   reads "not yet" again.)
        if (kMode == kModeDKDV) {
          if (!mbar_wait(bar + kBarYEmpty + 8 * (s & ~1), (use & 1u) ^ 1u, abort_flag)) return false;
        } else if ((idx & 1) == 0 && i >= 2) {
          if (!mbar_wait(bar + kBarSFull + 8 * ((i - 1) & 1), ((i - 1) >> 1) & 1, abort_flag)) return false;
        }
        const int hi = i / tiles_per_head;
        const int yt = y_lo + (i - hi * tiles_per_head);
        // dK/dV streams the query heads of this KV head; dQ streams the KV head of this query head
        const int hy = (kMode == kModeDKDV) ? query_head(hi) : hx / p.kv_group;
        const uint32_t full = bar + kBarYFull + 8 * s;
        const uint32_t dst = base + kSmemY + s * kYBytes;
        const int row = y_off + yt * kY;
        const bool first = (idx & 1) == 0;
        if (kMode == kModeDKDV && first) {
          mbar_arrive_expect_tx(full, kYBytes + 2 * kY * 4);
          const size_t vec = (static_cast<size_t>(b) * p.heads_q + hy) * p.lq_pad + static_cast<size_t>(yt) * kY;
          bulk_load_1d(base + kSmemVec + s * 1024, p.nlse2 + vec, kY * 4, full);
          bulk_load_1d(base + kSmemVec + s * 1024 + 512, p.ndelta + vec, kY * 4, full);
        } else {
          mbar_arrive_expect_tx(full, kYBytes);
        }
        const CUtensorMap* tm = first ? tmy1 : tmy2;
        tma_load_4d(dst, tm, full, 0, row, hy, bcoord);
        if (kD > 64) tma_load_4d(dst + kHalfBytes, tm, full, 64, row, hy, bcoord);
        else if (kY > kBoxRows) tma_load_4d(dst + kBoxBytes, tm, full, 0, row + kBoxRows, hy, bcoord);
    return true;
  };

  if (warp == kTmaWarp && lane == 0) {
    // descriptor fetches run under the barrier initialisation
    tma_prefetch_desc(tmx1);
    tma_prefetch_desc(tmy1);
    tma_prefetch_desc(tmx2);
    tma_prefetch_desc(tmy2);
    mbar_init(bar + kBarXFull, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar + kBarYFull + 8 * s, 1);
      mbar_init(bar + kBarYEmpty + 8 * s, 1);
    }
    mbar_init(bar + kBarSFull, 1);
    mbar_init(bar + kBarSFull + 8, 1);
    mbar_init(bar + kBarDFull, 1);
    mbar_init(bar + kBarDFree, kComputeWarps);  // one arrival per compute warp
    mbar_init(bar + kBarPFull, kComputeWarps);
    mbar_init(bar + kBarPFull + 8, kComputeWarps);
    mbar_init(bar + kBarP1Full, kComputeWarps);
    mbar_init(bar + kBarP1Full + 8, kComputeWarps);
    mbar_init(bar + kBarWFree, 1);
    mbar_init(bar + kBarWFree + 8, 1);
    mbar_init(bar + kBarSIssued, 1);
    mbar_init(bar + kBarEpiFull, kComputeWarps);
    mbar_init(bar + kBarAccFull, 1);
    *abort_flag = 0;
    fence_mbar_init();
    if (n_items > 0) {
      mbar_arrive_expect_tx(bar + kBarXFull, 2 * kXBytes);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const CUtensorMap* tm = x == 0 ? tmx1 : tmx2;
        const uint32_t dst = base + kSmemX + x * kXBytes;
        tma_load_4d(dst, tm, bar + kBarXFull, 0, x_row, hx, bcoord);
        if (kD > 64) tma_load_4d(dst + kHalfBytes, tm, bar + kBarXFull, 64, x_row, hx, bcoord);
        else tma_load_4d(dst + kBoxBytes, tm, bar + kBarXFull, 0, x_row + kBoxRows, hx, bcoord);
      }
    }
    if (kMode == kModeDKDV) {
      wait_for_previous_grid();
      if (!kPair) launch_dependents();
    }
    for (int idx = 0; idx < kPreloaded && idx < 2 * n_items; ++idx) load_tile(idx);
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(base + kSmemBar + kSmemTmemPtr, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  const uint32_t t1 = tmem_base, t2 = tmem_base + kY, acc1 = tmem_base + 2 * kY, acc2 = tmem_base + 2 * kY + kD;
#ifdef SDPA_BWD_STAMPS
  const long long t_start = clock64();
  // a long-running block of batch 0, head 0 (non-causal: any; causal: the heaviest)
  const bool stamp_on = p.stamps != nullptr && b == 0 && hx == 0 &&
                        xb == ((kMode == kModeDKDV) ? 0 : order.ranks - 1) && (lane == 0) &&
                        (warp == 0 || warp == 4 || warp == kScoreWarp || warp == kAccWarp);
#endif

  if (warp >= kTmaWarp) {
    if constexpr (kY == 64) reg_decrease<kRegsOther>();
    if (warp == kTmaWarp) {
      // ------------------------------------------------------------------ TMA producer (rest of the ring)
      if (n_items > 0 && elect_one()) {
        for (int idx = kPreloaded; idx < 2 * n_items; ++idx)
          if (!load_tile(idx)) break;
        drain_after_abort(abort_flag);
      }
    } else if (warp == kScoreWarp || warp == kAccWarp) {
      // ------------------------------------------------------------------ MMA issuers
      // One thread needs ~50-65 cycles to issue an MMA and ~70 for every barrier wait or commit, about
      // as long as the tensor pipe needs to execute it, and an item has 24 (dQ) or 32 (dK/dV) MMAs
      // plus half a dozen waits: a single issuer is the bottleneck. So two threads issue:
      //   kScoreWarp the score GEMMs   S = X1 Y1^T, dP = X2 Y2^T            (operands in shared memory)
      //   kAccWarp   the accumulations dV += P^T dO, dK += dS^T Q / dQ += dS K (A operand in TMEM)
      // What the in-order pipe would guarantee between the two groups is a barrier here: `W free`
      // (committed behind an item's accumulation MMAs; the score warp waits for it before a score GEMM
      // overwrites that item's P / dS buffer). There is one per item parity, so that the barrier a wait
      // looks at cannot be a whole phase further on: its next phase belongs to item i+2, whose scores
      // only exist after this wait.
      if (n_items > 0 && elect_one()) {
        // Where the score GEMMs of item i land:
        //   dK/dV: S(i) in T[i&1], dP(i) in T[(i&1)^1]. The compute warpgroups put BOTH 16-bit results
        //          (P and dS) into the S buffer, so the dP buffer is free once it has been read and
        //          takes S(i+1) right away; dP(i+1) goes into the S buffer behind the accumulations.
        //   dQ:    ACC2 is unused, so S alternates between T1 and ACC2 and dP always uses T2: S(i+2)
        //          follows the accumulation of item i, dP(i+1) goes out as soon as dP(i) is read.
        // Either way the next item's scores and exponentials run under this item's accumulation.
        // operand descriptors hold 18 bits of the address; in a cluster the bits above say which CTA it belongs to
        const uint32_t op_base = kSplit ? base & 0x3ffffu : base;
        const uint32_t x1 = op_base + kSmemX, x2 = op_base + kSmemX + kXBytes;
        auto s_buf = [&](int i) { return kMode == kModeDKDV ? ((i & 1) ? t2 : t1) : ((i & 1) ? acc2 : t1); };
        auto d_buf = [&](int i) { return kMode == kModeDKDV ? ((i & 1) ? t1 : t2) : t2; };
        auto s_bar = [&](int i) { return bar + kBarSFull + (kMode == kModeDQ ? 8 * (i & 1) : 0); };
        // ring position of tile 2i, kept incrementally (no division in the issue loop): slot = (2i) mod
        // kStages, lap = (2i) / kStages. Tiles 2i + k, k < kStages, follow from it with one wrap.
        // dQ splits its five slots into a K ring (slots 0-2) and a V ring (slots 3-4): a K tile lives
        // from its score GEMM to its accumulation GEMM two items later, a V tile only for one GEMM, so a
        // shared round-robin would free the slot V(i+1) needs too late to hide the load latency.
        int ring_slot = 0, ring_lap = 0;  // dK/dV: position of tile 2i; dQ: i mod 3 and i / 3
        int item = 0;
        auto pos = [&](int k, int& slot, int& lap) {
          if (kMode == kModeDKDV) {
            slot = ring_slot + k;
            lap = ring_lap;
            if (slot >= kStages) { slot -= kStages; ++lap; }
          } else if ((k & 1) == 0) {  // K(item + k/2)
            slot = ring_slot + (k >> 1);
            lap = ring_lap;
            if (slot >= 3) { slot -= 3; ++lap; }
          } else {  // V(item + k/2)
            const int j = item + (k >> 1);
            slot = 3 + (j & 1);
            lap = j >> 1;
          }
        };
        auto advance = [&]() {
          ++item;
          if (kMode == kModeDKDV) {
            ring_slot += 2;
            if (ring_slot >= kStages) { ring_slot -= kStages; ++ring_lap; }
          } else if (++ring_slot == 3) {
            ring_slot = 0;
            ++ring_lap;
          }
        };
        auto y_slot_k = [&](int k) { int sl, lp; pos(k, sl, lp); return op_base + kSmemY + sl * kYBytes; };
        auto y_wait_k = [&](int k) { int sl, lp; pos(k, sl, lp); return mbar_wait(bar + kBarYFull + 8 * sl, lp & 1, abort_flag); };
        auto y_free_k = [&](int k) { int sl, lp; pos(k, sl, lp); umma_commit(bar + kBarYEmpty + 8 * sl); };
        bool ok = true;
        if (warp == kScoreWarp) {
          // ---------------- score GEMMs
#ifdef SDPA_BWD_STAMPS
          if (stamp_on) p.stamps[((kMode * 4 + 2) * 24 + 23) * 8 + 0] = static_cast<float>(t_start - t_entry);
#endif
          ok = mbar_wait(bar + kBarXFull, 0, abort_flag) && y_wait_k(0);
          BWD_STAMP(2, 23, 1);
          if (ok) {
            tc_fence_after_sync();
            issue_xyT<kD, kF16, kY>(s_buf(0), x1, y_slot_k(0));
            umma_commit(s_bar(0));
          }
          BWD_STAMP(2, 23, 2);
          ok = ok && y_wait_k(1);
          if (ok) {
            tc_fence_after_sync();
            issue_xyT<kD, kF16, kY>(d_buf(0), x2, y_slot_k(1));
            umma_commit(bar + kBarDFull);
          }
          if (kMode == kModeDQ && ok && n_items > 1) {
            ok = y_wait_k(2);
            if (ok) {
              tc_fence_after_sync();
              issue_xyT<kD, kF16, kY>(s_buf(1), x1, y_slot_k(2));
              umma_commit(s_bar(1));
            }
          }
          for (int i = 0; ok && i < n_items; ++i, advance()) {
            const uint32_t sbuf = s_buf(i);
            const bool more = i + 1 < n_items;
            BWD_STAMP(2, i, 0);
            // dP(i) has left TMEM once all compute warps have read it
            ok = mbar_wait(bar + kBarDFree, i & 1, abort_flag);
            if (!ok) break;
            BWD_STAMP(2, i, 1);
            if (kMode == kModeDKDV) {
              if (!more) {
                mbar_arrive(bar + kBarSIssued);
                continue;
              }
              ok = y_wait_k(2);
              if (!ok) break;
              tc_fence_after_sync();
              issue_xyT<kD, kF16, kY>(d_buf(i), x1, y_slot_k(2));  // S(i+1) into the buffer dP(i) has just left
              umma_commit(s_bar(i + 1));
              // S(i+1) is what the compute warps wait for; dK(i) is not urgent. The other issuer holds
              // dK(i) back until this arrival, so the two GEMMs do not share the pipe MMA by MMA.
              mbar_arrive(bar + kBarSIssued);
              BWD_STAMP(2, i, 2);
              ok = mbar_wait(bar + kBarWFree + 8 * (i & 1), (i >> 1) & 1, abort_flag) && y_wait_k(3);
              if (!ok) break;
              BWD_STAMP(2, i, 3);
              tc_fence_after_sync();
              issue_xyT<kD, kF16, kY>(sbuf, x2, y_slot_k(3));  // dP(i+1) into the buffer P(i), dS(i) have left
              umma_commit(bar + kBarDFull);
              BWD_STAMP(2, i, 4);
            } else {
              if (more) {
                ok = y_wait_k(3);
                if (!ok) break;
                tc_fence_after_sync();
                issue_xyT<kD, kF16, kY>(t2, x2, y_slot_k(3));  // dP(i+1)
                umma_commit(bar + kBarDFull);
              }
              BWD_STAMP(2, i, 2);
              if (i + 2 < n_items) {
                ok = mbar_wait(bar + kBarWFree + 8 * (i & 1), (i >> 1) & 1, abort_flag) && y_wait_k(4);
                if (!ok) break;
                BWD_STAMP(2, i, 3);
                tc_fence_after_sync();
                issue_xyT<kD, kF16, kY>(sbuf, x1, y_slot_k(4));  // S(i+2) into the buffer dS(i) has left
                umma_commit(s_bar(i + 2));
                BWD_STAMP(2, i, 4);
              }
            }
          }
        } else {
          // ---------------- accumulation GEMMs
          ok = mbar_wait(bar + kBarXFull, 0, abort_flag);
          for (int i = 0; ok && i < n_items; ++i, advance()) {
            const uint32_t y1 = y_slot_k(0), y2 = y_slot_k(1);
            const uint32_t sbuf = s_buf(i);
            // the tiles have landed long ago (the other issuer has used them); this wait makes the
            // copies visible to this thread's MMAs as well
            ok = y_wait_k(0) && (kMode == kModeDQ || y_wait_k(1));
            if (!ok) break;
            if (kMode == kModeDKDV) {
              // dV needs P only, which is stored a whole dS pass before the item is complete
              ok = mbar_wait(bar + kBarP1Full + 8 * (i & 1), (i >> 1) & 1, abort_flag);
              if (!ok) break;
              tc_fence_after_sync();
              issue_wy<kD, kF16, kY>(acc1, sbuf, y2, i > 0);  // dV += P^T dO
            }
            BWD_STAMP(3, i, 0);
            ok = mbar_wait(bar + kBarPFull + 8 * (i & 1), (i >> 1) & 1, abort_flag);
            if (!ok) break;
            BWD_STAMP(3, i, 1);
            tc_fence_after_sync();
            if (kMode == kModeDKDV) {
              ok = mbar_wait(bar + kBarSIssued, i & 1, abort_flag);
              if (!ok) break;
              issue_wy<kD, kF16, kY>(acc2, sbuf + kC / 2, y1, i > 0);  // dK += dS^T Q
              y_free_k(0);  // releases the slot pair Q(i), dO(i)
            } else {
              issue_wy<kD, kF16, kY>(acc1, sbuf + kC / 2, y1, i > 0);  // dQ += dS K
            }
            umma_commit(bar + kBarWFree + 8 * (i & 1));
            if (i == n_items - 1) umma_commit(bar + kBarAccFull);
            BWD_STAMP(3, i, 2);
            if (i == 0) BWD_STAMP(3, 23, 0);
            if (i == n_items - 1) BWD_STAMP(3, 23, 1);
          }
        }
      }
    }
    if constexpr (kSplit) {  // the compute warps sum over the cluster
      cluster_sync();
      cluster_sync();
    }
  } else {
    // ------------------------------------------------------------------ compute warpgroups
    if constexpr (kY == 64) reg_increase<kRegsCompute>();
    // warps 0-3 own the first kC streamed columns of every stationary row, warps 4-7 the others
    const int half = warp >> 2;
    const int r = (warp & 3) * 32 + lane;  // stationary row in the tile = TMEM lane
    const int xr = x0 + r;                 // key index (dK/dV) or query index (dQ) within the sequence
    const uint32_t lane_base = (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * kC;
    const float c = p.scale_log2;
    bool ok = true;
    float my_nlse2 = 0.f, my_ndelta = 0.f;
    if (kMode == kModeDQ) {
      if (kPair) wait_for_previous_grid();  // the pre-pass; a dQ kernel of its own starts behind a grid that has waited for it
      const size_t vec = (static_cast<size_t>(b) * p.heads_q + hx) * p.lq_pad + xr;
      my_nlse2 = p.nlse2[vec];
      my_ndelta = p.ndelta[vec];
    }
    // dK/dV with a dQ GEMM behind it: the dS tile of the next item. One running register, since more of them spill
    uint32_t ds_tile = 0;
    if (kMode == kModeDKDV && kDsCall && p.ds.data != nullptr) {
      wait_for_previous_grid();  // DsTiles::seq_base comes from the pre-pass
      ds_tile = ds_head(p.ds, b, query_head(0), p.heads_q, len_q, len_k, p.is_causal != 0).tile(y_lo, xb);
    }
    for (int i = 0; i < n_items; ++i) {
      const int s = (2 * i) % kStages;  // ring slot of Y1(i), which carries the per-query vectors
      const int hi = i / tiles_per_head;
      const int y0 = (y_lo + (i - hi * tiles_per_head)) * kY;
      const uint32_t sbuf = (kMode == kModeDKDV ? ((i & 1) ? t2 : t1) : ((i & 1) ? acc2 : t1)) + lane_base;
      const uint32_t dbuf = (kMode == kModeDKDV ? ((i & 1) ? t1 : t2) : t2) + lane_base;
      BWD_STAMP(half, i, 0);
      // keep bits of this thread's kC (row, column) pairs, in flight under the waits below
      uint2 keep = make_uint2(0u, 0u);
      if constexpr (kDrop) {
        const uint32_t* words =
            (kMode == kModeDQ)
                ? p.keep_rows + (p.cu_q != nullptr ? static_cast<size_t>(hx) * p.keep_q_rows + q_off + xr
                                                   : static_cast<size_t>(b * p.heads_q + hx) * p.keep_q_rows + xr) *
                                    (p.keep_lk_pad >> 5)
                : p.keep_cols + (p.cu_q != nullptr
                                     ? static_cast<size_t>(query_head(hi)) * p.keep_k_rows + k_off + xr
                                     : static_cast<size_t>(b * p.heads_q + query_head(hi)) * p.keep_k_rows + xr) *
                                    (p.keep_lq_pad >> 5);
        if constexpr (kC == 64) keep = *reinterpret_cast<const uint2*>(words + ((y0 + half * kC) >> 5));
        else keep.x = words[(y0 + half * kC) >> 5];
      }
      uint32_t key_bias_raw = 0u;  // dK/dV: this key's value; dQ: the values of two of the kC keys
      if constexpr (kBias == kKeyBias) {
        const uint16_t* head = p.bias + b * p.bias_batch_stride + (kMode == kModeDQ ? hx : query_head(hi)) * p.bias_head_stride;
        const int key = y0 + half * kC + 2 * lane;
        if (kMode == kModeDQ && 2 * lane < kC && key < len_k) key_bias_raw = *reinterpret_cast<const uint32_t*>(head + key);
        if (kMode == kModeDKDV && xr < len_k) key_bias_raw = head[xr];
      }
      if constexpr (kBias == kFullBias) {
        // the next item's bias values of this thread's row: into L2 now (dQ: 128 contiguous bytes of the query
        // row; dK/dV: 64 query rows, two per lane, 64 bytes each around this warp's keys)
        if (i + 1 < n_items && xr < len_x) {
          const int hn = (i + 1) / tiles_per_head;
          const int cn = (y_lo + (i + 1 - hn * tiles_per_head)) * kY + half * kC;
          if (kMode == kModeDQ) {
            const uint16_t* nx = p.bias + b * p.bias_batch_stride + hx * p.bias_head_stride +
                                 static_cast<int64_t>(xr) * p.bias_row_stride + cn;
            if (cn < len_k) {  // only addresses inside the row
              prefetch_l2(nx);
              prefetch_l2(nx + min(kC - 1, len_k - 1 - cn));
            }
          } else {
            if (p.bias_t != nullptr) {
              const uint16_t* nx = p.bias_t + b * p.bias_t_batch_stride + query_head(hn) * p.bias_t_head_stride +
                                   static_cast<int64_t>(xr) * p.bias_t_row_stride + cn;
              if (cn < len_q) {
                prefetch_l2(nx);
                prefetch_l2(nx + min(kC - 1, len_q - 1 - cn));
              }
            } else {
              const uint16_t* nx = p.bias + b * p.bias_batch_stride + query_head(hn) * p.bias_head_stride + xr;
              const int q = 2 * lane < kC ? cn + 2 * lane : len_q;
              if (q < len_q) prefetch_l2(nx + static_cast<int64_t>(q) * p.bias_row_stride);
              if (q + 1 < len_q) prefetch_l2(nx + static_cast<int64_t>(q + 1) * p.bias_row_stride);
            }
          }
        }
      }
      // This item's bias values where they are contiguous for this thread (dQ: its query row; dK/dV: its key's row
      // of the transposed copy): eight 16-byte loads issued before the waits, so their latency passes under the
      // score GEMM. A chunk that starts past the end is skipped (zeros); one that straddles it reads row padding.
      uint4 bw[kBias == kFullBias ? kC / 8 : 1];
      bool bias_in_regs = false;
      if constexpr (kBias == kFullBias) {
        const int col0 = y0 + half * kC;
        const uint16_t* vrow = nullptr;
        int vlen = 0;
        if (kMode == kModeDQ) {
          vrow = p.bias + b * p.bias_batch_stride + hx * p.bias_head_stride + static_cast<int64_t>(xr) * p.bias_row_stride;
          vlen = len_k;
        } else if (p.bias_t != nullptr) {
          vrow = p.bias_t + b * p.bias_t_batch_stride + query_head(hi) * p.bias_t_head_stride +
                 static_cast<int64_t>(xr) * p.bias_t_row_stride;
          vlen = len_q;
        }
        bias_in_regs = vrow != nullptr;
        if (bias_in_regs) {
#pragma unroll
          for (int ch = 0; ch < kC / 8; ++ch) {
            bw[ch] = make_uint4(0u, 0u, 0u, 0u);
            if (xr < len_x && col0 + ch * 8 < vlen) bw[ch] = *reinterpret_cast<const uint4*>(vrow + col0 + ch * 8);
          }
        }
      }
      // `ok` is made warp-uniform after every wait: the warp-level arrivals below need all 32 lanes
      ok = mbar_wait(bar + kBarSFull + (kMode == kModeDQ ? 8 * (i & 1) : 0), (kMode == kModeDQ ? (i >> 1) : i) & 1,
                     abort_flag);
      if (kMode == kModeDKDV) {
        // the per-query vectors arrive with the stage's bulk copies; observe that barrier directly
        ok = ok && mbar_wait(bar + kBarYFull + 8 * s, ((2 * i) / kStages) & 1, abort_flag);
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      BWD_STAMP(half, i, 1);
      const float* vec_nlse = reinterpret_cast<const float*>(smem + kSmemVec + s * 1024) + half * kC;
      const float* vec_ndelta = vec_nlse + 128;
      // visibility of element (row xr, column y0 + j)
      //   dK/dV: key xr, query y0+j : visible iff xr <= y0 + j + off  <=>  j >= xr - off - y0
      //   dQ   : query xr, key y0+j : visible iff y0 + j <= xr + off and y0 + j < len_k
      int j_lo = 0, j_hi = kTile;
      if (kMode == kModeDKDV) {
        if (p.is_causal) j_lo = xr - causal_off - y0;
        // a row past the last key: its dS in the workspace must be zero (nothing else reads it, and the element mask costs time)
        if (kDsCall && p.ds.data != nullptr && xr >= len_x) j_lo = kTile;
      } else {
        j_hi = len_k - y0;
        if (p.is_causal) j_hi = min(j_hi, xr + causal_off + 1 - y0);
      }
      j_lo -= half * kC;  // relative to this thread's columns
      j_hi -= half * kC;

      // phase 1 (needs S only): P = exp2(S c - lse2), masked; its bf16 copy goes back at once
      float pr[kC];
      {
        uint32_t a[kC];
        tmem_ld_x32_at<0>(sbuf, a);
        if constexpr (kC > 32) tmem_ld_x32_at<32>(sbuf + 32, a);
        tmem_wait_ld();
        BWD_STAMP(half, i, 2);
        if constexpr (kBias == kFullBias) {
          // S <- S + bias / scale (then x = S c - lse2 as without bias)
          const int col0 = y0 + half * kC;
          if (bias_in_regs) {
#pragma unroll
            for (int ch = 0; ch < kC / 8; ++ch) {
              const uint32_t ww[4] = {bw[ch].x, bw[ch].y, bw[ch].z, bw[ch].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 b2 = unpack_16x2<kF16>(ww[e]);
                a[ch * 8 + 2 * e] = __float_as_uint(fmaf(b2.x, p.inv_scale, __uint_as_float(a[ch * 8 + 2 * e])));
                a[ch * 8 + 2 * e + 1] = __float_as_uint(fmaf(b2.y, p.inv_scale, __uint_as_float(a[ch * 8 + 2 * e + 1])));
              }
            }
          } else if (kMode == kModeDKDV && xr < len_x) {
            // no transposed copy: this key in kC consecutive query rows, as many two-byte loads (consecutive lanes on
            // consecutive keys)
            const uint16_t* bcol = p.bias + b * p.bias_batch_stride + query_head(hi) * p.bias_head_stride + xr;
#pragma unroll
            for (int j = 0; j < kC; ++j) {
              if (col0 + j < len_q) {
                const uint32_t raw = bcol[static_cast<int64_t>(col0 + j) * p.bias_row_stride];
                const float bv = unpack_16x2<kF16>(raw).x;
                a[j] = __float_as_uint(fmaf(bv, p.inv_scale, __uint_as_float(a[j])));
              }
            }
          }
        }
        constexpr float kLog2e = 1.4426950408889634f;
        float key_bias = 0.f, key_bias_log2 = 0.f;  // dK/dV
        uint32_t* key_bias_row = reinterpret_cast<uint32_t*>(smem + smem_key_bias_off(kMode, kD, kY) + warp * 128);  // dQ
        if constexpr (kBias == kKeyBias) {
          if (kMode == kModeDKDV) {
            key_bias = unpack_16x2<kF16>(key_bias_raw).x;
            key_bias_log2 = key_bias * kLog2e;
          } else {
            if (2 * lane < kC) key_bias_row[lane] = key_bias_raw;  // the previous item's values were read before this warp's last __syncwarp
            __syncwarp();
          }
        }
        // x = S c - lse2. kPolyOf4 of every four column pairs take their 2^x from the FMA pipe (exp2_poly3_x2). dQ: one; two already
        // cost issue slots. dK/dV: two, which shortens the chain of an item (step of B1 H8 L2048 D128 78.7 us, without any 82.0). None up to
        // head_dim 64: with two CTAs per SM one of four takes the same time (B8 H12 L1000 126, 126), and with one per SM, where two would save 0 to 6 %, the bits are to be the same. And none where dS goes through the workspace: those grids are full and run at the power
        // cap, where none to two take the same time (step of B8 H16 L2048 695, 694, 696 us, with dropout 858, 872, 870; B12 packed
        // 64 to 2048 tokens 369, 368, 364), and none is the most exact. Such a call without room for dS takes these two kernels, and its
        // bits must not tell: none here either, and the same roundings in both kernels (a key bias joins with one).
        constexpr int kPolyOf4 = kDsCall || kD == 64 ? 0 : kMode == kModeDQ ? 1 : 2;
#pragma unroll
        for (int j4 = 0; j4 < kC / 4; ++j4) {
          const float4 l = (kMode == kModeDKDV) ? read_vec4<kDrop>(vec_nlse + 4 * j4) : make_float4(my_nlse2, my_nlse2, my_nlse2, my_nlse2);
          uint2 kb = make_uint2(0u, 0u);
          if constexpr (kBias == kKeyBias && kMode == kModeDQ) kb = *reinterpret_cast<const uint2*>(key_bias_row + 2 * j4);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int j = 4 * j4 + 2 * h;
            float2 nl = h == 0 ? make_float2(l.x, l.y) : make_float2(l.z, l.w);
            if constexpr (kBias == kKeyBias) {
              const float2 kb2 = unpack_16x2<kF16>(h == 0 ? kb.x : kb.y), log2e = make_float2(kLog2e, kLog2e);
              nl = kMode == kModeDQ ? fma2(kb2, log2e, nl)
                   : kDsCall        ? fma2(make_float2(key_bias, key_bias), log2e, nl)
                                    : add2(nl, make_float2(key_bias_log2, key_bias_log2));
            }
            const float2 x = score_exponents<kDrop>(a[j], a[j + 1], c, nl);
            if (((j >> 1) & 3) < kPolyOf4) {
              const float2 e = exp2_poly3_x2(x);
              pr[j] = e.x;
              pr[j + 1] = e.y;
            } else {
              pr[j] = ex2_approx(x.x);
              pr[j + 1] = ex2_approx(x.y);
            }
          }
        }
        // only tiles on the causal diagonal or past the end of the keys need the element mask
        if (__any_sync(0xffffffffu, j_lo > 0 || j_hi < kC)) {
#pragma unroll
          for (int j = 0; j < kC; ++j) pr[j] = (j >= j_lo && j < j_hi) ? pr[j] : 0.f;
        }
        if (kMode == kModeDKDV) {
          uint32_t pw[kC / 2];
#pragma unroll
          for (int j2 = 0; j2 < kC / 2; ++j2) {
            if constexpr (kDrop) {
              const uint32_t word = j2 < 16 ? keep.x : keep.y;
              pw[j2] = pack_16x2<kF16>(kept(word, (2 * j2) & 31, pr[2 * j2]), kept(word, (2 * j2 + 1) & 31, pr[2 * j2 + 1]));
            } else {
              pw[j2] = pack_16x2<kF16>(pr[2 * j2], pr[2 * j2 + 1]);
            }
          }
          tmem_st_x16(sbuf, pw);
          if constexpr (kC > 32) tmem_st_x16(sbuf + 16, pw + 16);
          tmem_wait_st();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar + kBarP1Full + 8 * (i & 1));
        }
      }
      // phase 2 (needs dP): dS = P o (dP - delta) into the second half of this thread's columns
      BWD_STAMP(half, i, 3);
      ok = __all_sync(0xffffffffu, mbar_wait(bar + kBarDFull, i & 1, abort_flag));
      if (!ok) break;
      tc_fence_after_sync();
      BWD_STAMP(half, i, 4);
      uint32_t dw[kC / 2];
      {
        uint32_t d[kC];
        tmem_ld_x32_at<0>(dbuf, d);
        if constexpr (kC > 32) tmem_ld_x32_at<32>(dbuf + 32, d);
        tmem_wait_ld();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar + kBarDFree);  // the dP buffer may be overwritten
        BWD_STAMP(half, i, 5);
#pragma unroll
        for (int j4 = 0; j4 < kC / 4; ++j4) {
          const float4 l = (kMode == kModeDKDV) ? read_vec4<kDrop>(vec_ndelta + 4 * j4) : make_float4(my_ndelta, my_ndelta, my_ndelta, my_ndelta);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int j = 4 * j4 + 2 * h;
            const float2 nd = h == 0 ? make_float2(l.x, l.y) : make_float2(l.z, l.w);
            float2 e = make_float2(__uint_as_float(d[j]), __uint_as_float(d[j + 1]));
            if constexpr (kDrop) {  // M o dP / (1 - p) in the place of dP
              const uint32_t word = j < 32 ? keep.x : keep.y;
              e.x = pr[j] * fmaf(kept(word, j & 31, e.x), p.keep_scale, nd.x);
              e.y = pr[j + 1] * fmaf(kept(word, (j + 1) & 31, e.y), p.keep_scale, nd.y);
            } else {
              e = mul2(make_float2(pr[j], pr[j + 1]), add2(e, nd));
            }
            dw[j >> 1] = pack_16x2<kF16>(e.x, e.y);
          }
        }
        tmem_st_x16(sbuf + kC / 2, dw);
        if constexpr (kC > 32) tmem_st_x16(sbuf + kC / 2 + 16, dw + 16);
        if constexpr (kBias == kFullBias && kMode == kModeDQ) {
          // dbias = dS: this thread's keys of its query row, already packed for the dQ GEMM
          const int col0 = y0 + half * kC;
          if (p.dbias != nullptr && xr < len_x) {
            uint16_t* drow = p.dbias + b * p.dbias_batch_stride + hx * p.dbias_head_stride +
                             static_cast<int64_t>(xr) * p.dbias_row_stride + col0;
#pragma unroll
            for (int ch = 0; ch < kC / 8; ++ch)
              if (col0 + ch * 8 < len_k)
                *reinterpret_cast<uint4*>(drow + ch * 8) = make_uint4(dw[4 * ch], dw[4 * ch + 1], dw[4 * ch + 2], dw[4 * ch + 3]);
          }
        }
      }
      BWD_STAMP(half, i, 6);
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar + kBarPFull + 8 * (i & 1));
      BWD_STAMP(half, i, 7);
      if (kMode == kModeDKDV && kDsCall && p.ds.data != nullptr) {
        // dS for the dQ GEMM: 16 bytes (8 queries) per store, 512 contiguous bytes per warp. Behind the arrival, so that the
        // dK GEMM does not wait for the stores to issue. Without a hint to L2 (see bwd_ds_gemm_sm100.cu)
        if (ds_tile < p.ds.capacity) {
          uint4* dst = ds_group(p.ds, ds_tile, half * 8, r);
#pragma unroll
          for (int ch = 0; ch < kC / 8; ++ch)
            dst[ch * kDsTile] = make_uint4(dw[4 * ch], dw[4 * ch + 1], dw[4 * ch + 2], dw[4 * ch + 3]);
        }
        // past this row of tiles; behind the last one the next head's tiles begin
        const DsHead rows{0, (len_k + kTile - 1) / kTile, ds_shift(len_q, len_k, p.is_causal != 0)};
        ds_tile += min(max(y0 / kTile + rows.shift, 0), rows.key_tiles);
        if (i + 1 == (hi + 1) * tiles_per_head) ds_tile += rows.tile(y_lo, 0);
      }
    }

    // ---- epilogue: accumulators -> scale -> 16-bit -> global
    if (ok && n_items > 0) ok = mbar_wait(bar + kBarAccFull, 0, abort_flag);
    BWD_STAMP(half, 23, 0);
    if constexpr (kSplit) {
      // this CTA's part, fp32, for the sum over the cluster: 16 bytes (4 columns) per row, [column / 4][128 rows]; dV where K and V were, dK in
      // the ring, which is idle by now too
      if (ok) {
        tc_fence_after_sync();
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          float4* part = reinterpret_cast<float4*>(smem + (which == 0 ? kSmemX : kSmemY)) + r;
#pragma unroll
          for (int cc = 0; cc < kD / 64; ++cc) {
            const int col = half * (kD / 2) + cc * 32;
            uint32_t v[32];
            if (n_items > 0) {
              tmem_ld_x32((which == 0 ? acc1 : acc2) + (lane_base - half * kC) + col, v);
              tmem_wait_ld();
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
              part[(col / 4 + j) * kTile] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]),
                                                        __uint_as_float(v[4 * j + 3]));
          }
        }
      }
      // Sum over the cluster: every CTA takes its share of the rows out of all parts, in the order of the ranks. A CTA that has given up takes
      // part in the barriers.
      cluster_sync();
      const int rows = kTile / p.split;  // a multiple of 16
      for (int e = threadIdx.x; e < rows * (kD / 16) * 2; e += kComputeWarps * 32) {
        const int row = cluster_rank * rows + e % rows, chunk = e / rows;  // 16 columns of dV or dK
        const int which = chunk / (kD / 16), col = chunk % (kD / 16) * 16;
        const uint32_t part = base + (which == 0 ? kSmemX : kSmemY) + (col / 4 * kTile + row) * 16;
        float4 sum[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j] = cluster_ld_f32x4(part + j * kTile * 16, 0);
        for (int other = 1; other < p.split; ++other) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 x = cluster_ld_f32x4(part + j * kTile * 16, other);
            sum[j] = make_float4(sum[j].x + x.x, sum[j].y + x.y, sum[j].z + x.z, sum[j].w + x.w);
          }
        }
        if (x0 + row >= len_x) continue;
        const float mul = which == 1 ? p.scale : kDrop ? p.keep_scale : 1.f;
        const int64_t row_stride = which == 0 ? p.dv_row_stride : p.dk_row_stride;
        uint16_t* dst = which == 0 ? p.dv + hx * p.dv_head_stride : p.dk + hx * p.dk_head_stride;
        dst += (p.cu_q != nullptr ? k_off + x0 + row : static_cast<int64_t>(x0 + row)) * row_stride + col;
        if (p.cu_q == nullptr) dst += b * (which == 0 ? p.dv_batch_stride : p.dk_batch_stride);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (col + 8 * j >= p.head_dim) break;
          const float4 lo = sum[2 * j], hi = sum[2 * j + 1];
          *reinterpret_cast<uint4*>(dst + 8 * j) = make_uint4(pack_16x2<kF16>(lo.x * mul, lo.y * mul), pack_16x2<kF16>(lo.z * mul, lo.w * mul),
                                                              pack_16x2<kF16>(hi.x * mul, hi.y * mul), pack_16x2<kF16>(hi.z * mul, hi.w * mul));
        }
      }
      cluster_sync();  // the others have read this CTA's part
    } else if (ok) {
      tc_fence_after_sync();
      const bool valid = xr < len_x;
      // A whole 128-row tile leaves through shared memory and TMA stores (the ring slots are idle by
      // now): coalesced and asynchronous, where row-wise stores from registers - 128 bytes per thread,
      // every lane on another row - kept the load/store unit busy for ~4000 cycles per CTA. Dense
      // tensors are clipped by the tensor map; a packed (varlen) tile that ends inside its sequence's
      // last rows would spill into the next sequence and is written row by row instead.
      const bool use_tma = (p.cu_q == nullptr) || (x0 + kTile <= len_x);
      const int n_out = (kMode == kModeDKDV) ? 2 : 1;
      constexpr int kColumns = kD / 2;  // head_dim columns per warpgroup
#pragma unroll
      for (int which = 0; which < n_out; ++which) {
        uint16_t* dst;
        float mul;
        uint32_t acc;
        if (kMode == kModeDQ) {
          dst = p.dq + ((p.cu_q != nullptr) ? static_cast<int64_t>(q_off + xr) * p.dq_row_stride
                                            : b * p.dq_batch_stride + static_cast<int64_t>(xr) * p.dq_row_stride) +
                hx * p.dq_head_stride;
          mul = p.scale;
          acc = acc1;
        } else if (which == 0) {
          dst = p.dv + ((p.cu_q != nullptr) ? static_cast<int64_t>(k_off + xr) * p.dv_row_stride
                                            : b * p.dv_batch_stride + static_cast<int64_t>(xr) * p.dv_row_stride) +
                hx * p.dv_head_stride;
          mul = kDrop ? p.keep_scale : 1.f;
          acc = acc1;
        } else {
          dst = p.dk + ((p.cu_q != nullptr) ? static_cast<int64_t>(k_off + xr) * p.dk_row_stride
                                            : b * p.dk_batch_stride + static_cast<int64_t>(xr) * p.dk_row_stride) +
                hx * p.dk_head_stride;
          mul = p.scale;
          acc = acc2;
        }
#pragma unroll
        // this warpgroup converts its share of the head_dim columns
        for (int cc = 0; cc < kColumns / 32; ++cc) {
          uint32_t v[32];
          if (n_items > 0) {
            tmem_ld_x32(acc + (lane_base - half * kC) + half * kColumns + cc * 32, v);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0u;
          }
          uint4 w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            w[j].x = pack_16x2<kF16>(__uint_as_float(v[8 * j + 0]) * mul, __uint_as_float(v[8 * j + 1]) * mul);
            w[j].y = pack_16x2<kF16>(__uint_as_float(v[8 * j + 2]) * mul, __uint_as_float(v[8 * j + 3]) * mul);
            w[j].z = pack_16x2<kF16>(__uint_as_float(v[8 * j + 4]) * mul, __uint_as_float(v[8 * j + 5]) * mul);
            w[j].w = pack_16x2<kF16>(__uint_as_float(v[8 * j + 6]) * mul, __uint_as_float(v[8 * j + 7]) * mul);
          }
          const int col = half * kColumns + cc * 32;  // first of this thread's 32 columns
          if (use_tma) {
            // output tile `which` is staged in the ring: 64-column halves of 128-byte rows
            // in the 128-byte-swizzled layout the tensor map expects
            uint8_t* row = smem + kSmemY + which * kXBytes + (col >> 6) * kHalfBytes + r * 128;
            const int chunk0 = (col & 63) >> 3;
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(row + (((chunk0 + j) ^ (r & 7)) << 4)) = w[j];
          } else if (valid) {
            uint4* o4 = reinterpret_cast<uint4*>(dst + col);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col + 8 * j < p.head_dim) o4[j] = w[j];
          }
        }
      }
      if (use_tma) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar + kBarEpiFull);
        if (threadIdx.x == 0) {
          if (mbar_wait(bar + kBarEpiFull, 0, abort_flag)) {
            const int row0 = ((kMode == kModeDKDV) ? k_off : q_off) + x0;
#pragma unroll
            for (int which = 0; which < n_out; ++which) {
              const CUtensorMap* tm = (which == 0) ? &tm_o1 : &tm_o2;
#pragma unroll
              for (int ht = 0; ht < kD / 64; ++ht)
                tma_store_4d(tm, base + kSmemY + which * kXBytes + ht * kHalfBytes, ht * 64, row0, hx, bcoord);
            }
            tma_store_commit();
            tma_store_wait_read();  // the shared memory must outlive the stores' reads of it
          }
        }
      }
    }
  }

  if (warp < kTmaWarp) BWD_STAMP(warp >> 2, 23, 1);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (warp == 0) BWD_STAMP(0, 23, 2);
  if (threadIdx.x == 0 && *abort_flag != 0) atomicExch(p.status, SDPA_B200_DEVICE_TIMEOUT);
  // the dQ grid overlaps the tail of the dK/dV grid: it must not be the first of the two to complete
  if (kMode == kModeDQ && threadIdx.x == 0) wait_for_previous_grid();
}

template <int kMode, int kD, bool kF16, bool kDrop, int kBias, bool kDsCall, bool kSplit, int kY>
__global__ void __launch_bounds__(kThreads<kY>, kY == 64 ? 2 : 1)
bwd_tile_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_o1, const __grid_constant__ CUtensorMap tm_o2,
                const __grid_constant__ BwdKernelParams p) {
  tile_cta<kMode, kD, kF16, kDrop, kBias, kDsCall, kSplit, kY, false>(tm_q, tm_k, tm_v, tm_do, tm_o1, tm_o2, p, p.order, p.heads_x, blockIdx.x);
}

// Both kernels in one launch: the dK/dV blocks, then the dQ blocks.
struct DqGrid {
  BlockOrder order;
  int heads_x;
  int first;  // block of the grid
};
template <int kD, bool kF16, bool kDrop, int kBias, int kY>
__global__ void __launch_bounds__(kThreads<kY>, kY == 64 ? 2 : 1)
bwd_tile_kernel_pair(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ CUtensorMap tm_dv, const __grid_constant__ CUtensorMap tm_dk,
                     const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ BwdKernelParams p, const DqGrid dq) {
  const int block = static_cast<int>(blockIdx.x) - dq.first;
  if (block < 0)
    tile_cta<kModeDKDV, kD, kF16, kDrop, kBias, false, false, kY, true>(tm_q, tm_k, tm_v, tm_do, tm_dv, tm_dk, p, p.order, p.heads_x, blockIdx.x);
  else
    tile_cta<kModeDQ, kD, kF16, kDrop, kBias, false, false, kY, true>(tm_q, tm_k, tm_v, tm_do, tm_dq, tm_dq, p, dq.order, dq.heads_x, block);
}

// ndelta[row] = -sum_d dO[row,d] * O[row,d]; nlse2[row] = -lse[row] * log2(e);
// rows padded to lq_pad per (batch, head): padding rows get nlse2 = -inf, ndelta = 0.
struct PreParams {
  const uint16_t* out;
  const uint16_t* dout;
  const float* lse;
  float* nlse2;
  float* ndelta;
  const int32_t* cu_q;
  int64_t o_batch_stride, o_head_stride, o_row_stride;
  int64_t do_batch_stride, do_head_stride, do_row_stride;
  int seqlen_q, total_q, heads_q, lq_pad, head_dim;
  int block0;       // first block of rows of this launch
  float* dq_acc;    // fused kernel: its dQ accumulator, whose existing rows are cleared here; else null
  int dq_acc_rows;  // as in BwdKernelParams
  int32_t* ds_seq_base;  // packed, dS for a dQ GEMM: DsTiles::seq_base, written here; else null
  const int32_t* cu_k;
  int is_causal;
  PackedGrads grads;
};

// 16 bytes (8 elements) per thread and kD / 8 threads per row; a 256-thread block covers two passes of rows of the padded sequence. HBM-bound:
// all loads of a block, the logsumexp among them, are issued before the first use, and the rows' sums go through shared memory, so
// that a block has one memory latency instead of two and writes whole lines (with the logsumexp read behind the sums by one lane per row
// and four passes per block, 134 MB at B8 H16 L2048 D128 29.8 us; so 22.6, 5.9 TB/s; four passes 23.0, one 24.6).
template <int kD>
constexpr int kPreRows = 2 * 256 * 8 / kD;  // 64 or 32
constexpr int kMaxGridY = 65535;
// Blocks per SM: 32 registers dense, 40 packed. (Packed without the limit, above head_dim 64, 47 registers and five blocks: 12 sequences of 64 to 2048 tokens, 16 heads 20.6 us, so 18.5.)
template <bool kPacked>
constexpr int kPreBlocks = kPacked ? 6 : 8;
template <int kD, bool kF16, bool kPacked>
__global__ void __launch_bounds__(256, kPreBlocks<kPacked>) bwd_preprocess_kernel(const PreParams p) {
  if (kPacked && static_cast<int>(blockIdx.x) == p.heads_q) {
    clear_uncovered_rows(p.grads, p.heads_q);
    return;
  }
  if (threadIdx.x == 0) launch_dependents();  // see bwd_tile_kernel
  constexpr int kRows = kPreRows<kD>, kPerPass = kRows / 2, kThreadsPerRow = kD / 8;
  __shared__ float sums[kRows];
  // heads vary fastest across the grid: with the usual [batch, row, head, dim] memory order the blocks
  // that run together then read neighbouring 256-byte pieces of the same rows
  const int h = blockIdx.x, b = blockIdx.z;
  const int col = threadIdx.x % kThreadsPerRow * 8;
  const int r_in_pass = threadIdx.x / kThreadsPerRow;
  int q_off = 0, len_q = p.seqlen_q;
  if (kPacked) {
    q_off = p.cu_q[b];
    len_q = p.cu_q[b + 1] - q_off;
  }
  if (kPacked && p.ds_seq_base != nullptr && h == 0 && blockIdx.y == 0 && p.block0 == 0) {
    write_seq_base(p.ds_seq_base, p.cu_q, p.cu_k, b, p.is_causal != 0);
  }
  // Packed: as many blocks per sequence as one of the mean length has (launch_bwd), which go on where there are more rows, up to the last row that a tile of the kernels
  // behind has; with blocks for the longest one in all of them half were empty (12 sequences of 64 to 2048 tokens, 16 heads, D128 25.3 us, so 18.5; 20 of 100 to 3000, D64 with the
  // accumulator 47.7, 46.1; one of 4096 among 7 of 16, D64 16.3, 7.9).
  const int rows = kPacked ? min((len_q + kTile - 1) / kTile * kTile, p.lq_pad) : p.lq_pad;
  for (int row0 = (p.block0 + blockIdx.y) * kRows; row0 < rows; row0 += gridDim.y * kRows) {
    uint4 ov[2], dv[2];
#pragma unroll
    for (int ps = 0; ps < 2; ++ps) {
      ov[ps] = make_uint4(0u, 0u, 0u, 0u);
      dv[ps] = make_uint4(0u, 0u, 0u, 0u);
      const int row = row0 + ps * kPerPass + r_in_pass;
      if (row < len_q && col < p.head_dim) {
        const int64_t at = (kPacked ? q_off : 0) + static_cast<int64_t>(row);
        const uint16_t* o = p.out + (kPacked ? 0 : b * p.o_batch_stride) + h * p.o_head_stride + at * p.o_row_stride + col;
        const uint16_t* dout = p.dout + (kPacked ? 0 : b * p.do_batch_stride) + h * p.do_head_stride + at * p.do_row_stride + col;
        ov[ps] = __ldcs(reinterpret_cast<const uint4*>(o));  // not read again, unlike dO
        dv[ps] = *reinterpret_cast<const uint4*>(dout);
      }
    }
    const int my_row = row0 + threadIdx.x;  // of the first kRows threads: the row whose values they write
    const bool have = threadIdx.x < kRows && my_row < len_q;
    float lse = 0.f;
    if (have)
      lse = kPacked ? p.lse[static_cast<size_t>(h) * p.total_q + q_off + my_row]
                    : p.lse[(static_cast<size_t>(b) * p.heads_q + h) * p.seqlen_q + my_row];
    if (kD == 64 && p.dq_acc != nullptr) {
      // 64 rows of an accumulator tile: per 4-column group 1 KB of consecutive floats, a thread per row. The stores need no
      // registers and go out under the loads above
      constexpr int groups = 16;
      const int row = row0 + (threadIdx.x & (kRows - 1));
      if (row < len_q) {
        const size_t acc_row = kPacked ? static_cast<size_t>(h) * p.dq_acc_rows + q_off + row
                                                 : (static_cast<size_t>(b) * p.heads_q + h) * p.lq_pad + row;
        float4* dst = reinterpret_cast<float4*>(p.dq_acc + (acc_row >> 7) * (static_cast<size_t>(groups) * 512)) + (acc_row & 127);
        for (int g = threadIdx.x / kRows; g < groups; g += 256 / kRows) dst[g * 128] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int ps = 0; ps < 2; ++ps) {
      const float2 o0 = unpack_16x2<kF16>(ov[ps].x), o1 = unpack_16x2<kF16>(ov[ps].y);
      const float2 o2 = unpack_16x2<kF16>(ov[ps].z), o3 = unpack_16x2<kF16>(ov[ps].w);
      const float2 d0 = unpack_16x2<kF16>(dv[ps].x), d1 = unpack_16x2<kF16>(dv[ps].y);
      const float2 d2 = unpack_16x2<kF16>(dv[ps].z), d3 = unpack_16x2<kF16>(dv[ps].w);
      float acc = (o0.x * d0.x + o0.y * d0.y) + (o1.x * d1.x + o1.y * d1.y) + (o2.x * d2.x + o2.y * d2.y) +
                  (o3.x * d3.x + o3.y * d3.y);
      // the threads of a row are consecutive lanes of one warp
#pragma unroll
      for (int off = kThreadsPerRow >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (col == 0) sums[ps * kPerPass + r_in_pass] = acc;
    }
    __syncthreads();
    if (threadIdx.x < kRows && my_row < p.lq_pad) {
      const size_t dst = (static_cast<size_t>(b) * p.heads_q + h) * p.lq_pad + my_row;
      p.nlse2[dst] = have ? lse * -1.4426950408889634f : -INFINITY;
      p.ndelta[dst] = have ? -sums[threadIdx.x] : 0.f;
    }
    if (!kPacked) break;
    __syncthreads();  // the sums have been read
  }
}

using TileKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                            const CUtensorMap, const CUtensorMap, const BwdKernelParams);

template <int kMode, bool kDrop, int kBias, bool kSplit, int kD, bool kDsCall, int kY>
TileKernel pick_tile_kernel(bool f16) {
  return f16 ? bwd_tile_kernel<kMode, kD, true, kDrop, kBias, kDsCall, kSplit, kY> : bwd_tile_kernel<kMode, kD, false, kDrop, kBias, kDsCall, kSplit, kY>;
}

template <int kMode, bool kDrop, int kBias, bool kSplit = false>
TileKernel pick_tile_kernel(int head_dim, bool f16, bool ds_call, bool wide) {
  if (head_dim <= 64) {
    if constexpr (!kSplit)
      if (wide) return pick_tile_kernel<kMode, kDrop, kBias, kSplit, 64, false, kTile>(f16);
    return pick_tile_kernel<kMode, kDrop, kBias, kSplit, 64, false, 64>(f16);
  }
  return ds_call ? pick_tile_kernel<kMode, kDrop, kBias, kSplit, 128, true, kTile>(f16) : pick_tile_kernel<kMode, kDrop, kBias, kSplit, 128, false, kTile>(f16);
}

template <int kMode, bool kDrop>
TileKernel pick_tile_kernel(BiasKind bias, int head_dim, bool f16, bool ds_call, bool wide) {
  if (bias == kKeyBias) return pick_tile_kernel<kMode, kDrop, kKeyBias>(head_dim, f16, ds_call, wide);
  return bias == kFullBias ? pick_tile_kernel<kMode, kDrop, kFullBias>(head_dim, f16, ds_call, wide)
                           : pick_tile_kernel<kMode, kDrop, kNoBias>(head_dim, f16, ds_call, wide);
}

template <int kMode>
TileKernel pick_tile_kernel(bool drop, BiasKind bias, int head_dim, bool f16, bool ds_call, bool wide) {
  return drop ? pick_tile_kernel<kMode, true>(bias, head_dim, f16, ds_call, wide)
              : pick_tile_kernel<kMode, false>(bias, head_dim, f16, ds_call, wide);
}

// `overlap_previous`: launch with programmatic stream serialization, so that this grid's CTAs may start as soon as
// every CTA of the kernel before it in the stream has signalled launch_dependents and an SM has room. Used for the dK/dV kernel
// behind the pre-pass, and for the dQ kernel, which needs nothing the dK/dV kernel writes: its CTAs fill the SMs the last, partly
// empty wave of dK/dV CTAs leaves idle. `wide`, up to head_dim 64: streamed tiles of 128 rows, one CTA per SM.
int launch_tile_kernel(int mode, int head_dim, bool f16, int grid, bool wide, cudaStream_t stream, const CUtensorMap& tm_q,
                       const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_do,
                       const CUtensorMap& tm_o1, const CUtensorMap& tm_o2, const BwdKernelParams& kp,
                       bool overlap_previous = false) {
  const bool drop = kp.keep_rows != nullptr;
  // the dK/dV kernel writes no bias gradient
  const BiasKind bias = kp.bias == nullptr                                                                    ? kNoBias
                        : kp.bias_row_stride == 0 && (mode == kModeDKDV || kp.dbias == nullptr) ? kKeyBias
                                                                                                              : kFullBias;
  const bool split = mode == kModeDKDV && kp.split > 1;
  TileKernel kernel = split ? (drop ? pick_tile_kernel<kModeDKDV, true, kNoBias, true>(head_dim, f16, kp.ds_call != 0, false)
                                    : pick_tile_kernel<kModeDKDV, false, kNoBias, true>(head_dim, f16, kp.ds_call != 0, false))
                      : mode == kModeDKDV ? pick_tile_kernel<kModeDKDV>(drop, bias, head_dim, f16, kp.ds_call != 0, wide)
                                        : pick_tile_kernel<kModeDQ>(drop, bias, head_dim, f16, kp.ds_call != 0, wide);
  const int dim = head_dim <= 64 ? 64 : 128, rows = dim == 64 && (split || !wide) ? 64 : kTile;  // the instance
  const uint32_t smem = smem_bytes_for(mode, dim, rows, bias == kKeyBias);
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) {
    set_error("backward: cudaFuncSetAttribute(%u bytes smem): %s", smem, cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(split ? grid * kp.split : grid);
  cfg.blockDim = dim3(rows == 64 ? kThreads<64> : kThreads<kTile>);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (overlap_previous) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (split) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = kp.split;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  err = cudaLaunchKernelEx(&cfg, kernel, tm_q, tm_k, tm_v, tm_do, tm_o1, tm_o2, kp);
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("backward %s: launch failed: %s", mode == kModeDKDV ? "dK/dV" : "dQ", cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  return SDPA_B200_OK;
}

using PairKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                            const CUtensorMap, const CUtensorMap, const BwdKernelParams, const DqGrid);
template <bool kDrop, int kBias>
PairKernel pick_pair_kernel(int head_dim, bool f16, bool wide) {
  if (head_dim > 64) return f16 ? bwd_tile_kernel_pair<128, true, kDrop, kBias, kTile> : bwd_tile_kernel_pair<128, false, kDrop, kBias, kTile>;
  if (wide) return f16 ? bwd_tile_kernel_pair<64, true, kDrop, kBias, kTile> : bwd_tile_kernel_pair<64, false, kDrop, kBias, kTile>;
  return f16 ? bwd_tile_kernel_pair<64, true, kDrop, kBias, 64> : bwd_tile_kernel_pair<64, false, kDrop, kBias, 64>;
}

// The dK/dV and the dQ kernel of a call without clusters, dS or a bias that depends on the query, as one launch behind the pre-pass.
int launch_tile_pair(int head_dim, bool f16, int grid_dkdv, int grid_dq, const DqGrid& dq, bool wide, cudaStream_t stream, const CUtensorMap& tm_q,
                     const CUtensorMap& tm_k, const CUtensorMap& tm_v, const CUtensorMap& tm_do, const CUtensorMap& tm_dv, const CUtensorMap& tm_dk,
                     const CUtensorMap& tm_dq, const BwdKernelParams& kp) {
  const bool key_bias = kp.bias != nullptr;
  PairKernel kernel = kp.keep_rows != nullptr ? (key_bias ? pick_pair_kernel<true, kKeyBias>(head_dim, f16, wide) : pick_pair_kernel<true, kNoBias>(head_dim, f16, wide))
                                              : (key_bias ? pick_pair_kernel<false, kKeyBias>(head_dim, f16, wide) : pick_pair_kernel<false, kNoBias>(head_dim, f16, wide));
  const int dim = head_dim <= 64 ? 64 : 128, rows = dim == 64 && !wide ? 64 : kTile;
  const uint32_t one = smem_bytes_for(kModeDKDV, dim, rows, key_bias), other = smem_bytes_for(kModeDQ, dim, rows, key_bias), smem = one > other ? one : other;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) {
    set_error("backward: cudaFuncSetAttribute(%u bytes smem): %s", smem, cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid_dkdv + grid_dq);
  cfg.blockDim = dim3(rows == 64 ? kThreads<64> : kThreads<kTile>);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  err = cudaLaunchKernelEx(&cfg, kernel, tm_q, tm_k, tm_v, tm_do, tm_dv, tm_dk, tm_dq, kp, dq);
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("backward dK/dV and dQ: launch failed: %s", cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  return SDPA_B200_OK;
}

int lq_padded(const sdpa_b200_params& p) { return ((p.max_seqlen_q + kTile - 1) / kTile) * kTile; }

}  // namespace

// Which kernels a call takes, with figures in us ("step": forward and backward in turn over seconds; the others the backward alone,
// calls back to back):
//  * up to one CTA per SM for the key blocks: the dK/dV and the dQ kernel side by side (bwd_tile_kernel twice). Whatever waits for
//    the dK/dV kernel waits for a whole chain of items while SMs are idle. (B1 H8 L2048 D128 step 85, through dS 95, fused 103; B4
//    H8/1 L4096 545, 564, 800; the other way round only where few key blocks meet many queries: B2 H32/8 L1024 unmasked 124, 112.)
//  * a bias gradient: the same two, since the dQ kernel, whose threads own query rows, writes it.
//  * head_dim 64, more key blocks, no bias, no fixed order asked for: the fused kernel where rows are long or query heads grouped, the two kernels
//    where clusters share a group of query heads (bwd_split) and where rows are short, since their two CTAs per SM hide set-up and epilogue, and with dropout, where the fused kernel reads keep
//    bits on its chain. (Step, fused | two kernels: B8 H16 L2048 471 | 476, B2 H16 L4096 unmasked 727 | 787, B8 H16 L1500 unmasked 485 | 505, packed
//    30 to 300 tokens, 32/8 heads 133 | 137; B16 H16 L1024 318 | 305, L500 131 | 121, B8 H12 L1000 unmasked 197 | 187, packed 100 to 600 tokens 203 | 192;
//    dropout B32 H12 L300 unmasked 208 | 180, B8 H16 L2000 693 | 675. Through dS, when its kernels had one CTA per SM: B8 H16 L2048 530.)
//  * head_dim 65 to 128, more key blocks: dS through the workspace and a GEMM for dQ (use_ds_backward). One pass over the scores where
//    the two kernels make two, and no reductions. (Step of B8 H16 L2048 695, two kernels 757, fused 752; with dropout 875, 940, 925;
//    B2 H16 L8192, in two passes, 2189, 2295, 2290; B16 H32 L512 310, 365, 360; D80 B8 H16 L2048 alone 438, 533, 545; grouped B8 H32/8 L2048 alone
//    860, 1100, 1130, B16 H16/4 L700 165, 208, 206.) The smallest of these grids, replayed from a graph: B3 H50 L128 alone 23.1, 22.3,
//    27.0, B2 H80 L256 45.3, 46.0, 53.8, grouped B2 H80/40 L256 41.1, 42.9, 43.0, with dropout 45.7, 47.3, 58.3.
// A packed call counts the key blocks of its grid, every sequence at the longest length, whether they have keys or not. The number
// of SMs is the B200's, not the current device's: workspace queries and launches must agree.
int64_t key_blocks(const sdpa_b200_params& p) {
  return static_cast<int64_t>(p.batch) * p.heads_kv * ((static_cast<int64_t>(p.max_seqlen_k) + kTile - 1) / kTile);
}
constexpr int64_t kSms = 148;

// Up to head_dim 64: streamed tiles of 128 rows, from the blocks of a launch and the longest chain of such items. With blocks for at most half of the SMs every block has a pair
// of SMs to itself, and with one per SM long chains are worth it still. (Backward alone, 64 rows | 128, us; up to 74 blocks: B1 H8 L1051 unmasked 30.7 | 23.8, B6 H8/1 L197
// unmasked 41.0 | 32.8, B2 H8 L453 20.5 | 16.4, B1 H16 L308 15.7 | 14.4; up to 148: B3 H32/8 L457 unmasked 57.2 | 47.6, B5 H16/4 L709 86.3 | 73.9, B1 H16 L656 causal, a chain of 6, 23.1 |
// 18.5; but chains of 5, 4, 3 and 1: B1 H16 L539 21.4 | 24.6, B2 H16 L475 21.5 | 23.9, B4 H12 L285 18.5 | 22.3, B7 H16 L75 12.6 | 14.4.)
bool wide_tiles(double blocks, int chain) { return blocks <= kSms / 2 || (blocks <= kSms && chain >= 6); }

// CTAs that share the query heads of a key block (calls without bias). One CTA sums a whole group, in a chain of group x query tiles items;
// where the longest chain is a multiple (the ratio below) of what an SM has to do on average, a cluster takes the heads in shares and sums
// its parts through shared memory. A packed call counts lengths spread between the mean and the longest. (Step in us, one CTA | two | four;
// packed, causal unless said. Up to head_dim 64, "one" the fused kernel where it would run: ratio 1, 3 sequences of 200 to 3000 tokens, 16/4
// heads, unmasked 402 | 377 | 363; 1, 8 of 64 to 2000, 16/4 331 | 295 | 331; 2.1, 16 of 64 to 2000, 8/1 374 | 321 | 296; 2.3, chain of 36, 4 of 64 to
// 1280, 32/8 132 | 122 | 137; 4.5, 4 of 64 to 1280, 16/4 121 | 93 | 83; rows of nearly one length, whose chains fill the SMs more evenly: 1.24,
// 2 of 1900 to 2000, 16/4, unmasked 260 | 225, and 1.4, 5 of 900 to 1700 191 | 184; but 1.18, 4 of 2000 to 2100 244 | 255; also 0.6, 8 of 500 to
// 1500, 32/8 374 | 404. Chains of less than 48 want a ratio of two there as well where the fused kernel is the other choice, which is the better one for them (but against one CTA per block, up to
// 148 of them: 1.2, chain of 24, 5 of 654, 16/4 backward alone 70 | 64): backward alone, 1.23, chain of 32, 32 of 197
// to 397, 64/8 165 | 184, 1.71, 24, 8 of 175 to 708, 32/8 80 | 88, 1.41, 44, 4 of 636 to 1336, 32/8 111 | 122; but 2.4, 30, 32 of 136 to 631, 12/2 97 | 94, and longer ones 1.25, 60, 10 of
// 385 to 1850 178 | 175, 1.1, 144, 32 of 328 to 2297, 8/1 486 | 388. D128: 2.3, 16 of 100 to 2500, 8/1 489 | 405 | 433; 4.6, 2 of 300 to 2000, 16/4 151 | 112 | 120; 8, 6 of 200 to 1500, 8/1
// 232 | 154 | 116, eight 152; but 1, 12 of 64 to 2048, 16/4 326 | 351, and 2.4, chain of 20, 8 of 64 to 700, 16/4, unmasked 103.5 | 108.5: a cluster
// waits for SMs that are free together and for its slowest part.)
int bwd_split(const sdpa_b200_params& p) {
  const int group = p.heads_q / p.heads_kv;
  const double query_tiles = (p.max_seqlen_q + kTile - 1) / kTile;
  const double mean_tiles = p.cu_seqlens_q != nullptr ? static_cast<double>(p.total_q) / p.batch / kTile : query_tiles;
  const double key_tiles = p.cu_seqlens_q != nullptr ? mean_tiles : (p.max_seqlen_k + kTile - 1) / kTile;
  const double items = static_cast<double>(p.batch) * p.heads_q * key_tiles * (mean_tiles + query_tiles) / 2 * (p.is_causal ? 0.5 : 1.0);
  const double ratio = group * query_tiles * kSms / (items > 1 ? items : 1);
  const bool narrow = p.head_dim <= 64;
  const double chain = group * query_tiles;
  if (p.bias != nullptr || chain < (narrow ? 24 : 32)) return 1;
  if (group % 4 == 0 && ratio >= (narrow ? (chain < 64 ? 3.0 : 2.0) : 6.0)) return 4;
  const bool or_fused = p.deterministic == 0 && key_blocks(p) > kSms;  // what the call would take instead
  return group % 2 == 0 && ratio >= (!narrow || (or_fused && chain < 48) ? 2.0 : mean_tiles < 0.75 * query_tiles ? 0.9 : 1.2) ? 2 : 1;
}

bool use_ds_backward(const sdpa_b200_params& p) {
  return p.head_dim > 64 && p.dbias == nullptr && key_blocks(p) > kSms;
}

bool use_fused_backward(const sdpa_b200_params& p) {
  const int longest = p.max_seqlen_q > p.max_seqlen_k ? p.max_seqlen_q : p.max_seqlen_k;
  const bool short_rows = p.heads_q == p.heads_kv && longest <= (p.dropout_p > 0.f ? 2048 : 1024);
  return p.head_dim <= 64 && p.deterministic == 0 && p.bias == nullptr && key_blocks(p) > kSms && !short_rows && bwd_split(p) == 1;
}

size_t bwd_vector_bytes(const sdpa_b200_params& p) {
  const size_t bytes = 2 * static_cast<size_t>(p.batch) * p.heads_q * lq_padded(p) * sizeof(float);
  return (bytes + 255) / 256 * 256;
}

// What a call needs: lse2 and delta, then the fp32 dQ accumulator of the fused kernel: for every call up to head_dim 64 without a bias
// that does not ask for a fixed order, whatever path its sizes take, so that one workspace serves calls that differ in sizes.
size_t bwd_workspace_min_bytes(const sdpa_b200_params& p) {
  const bool acc = p.head_dim <= 64 && p.deterministic == 0 && p.bias == nullptr;
  return bwd_vector_bytes(p) + (acc ? bwd_fused_workspace_bytes(p, lq_padded(p)) : 0);
}

// What it is best given: room for dS too. A call that is given less takes the two kernels.
size_t bwd_workspace_bytes(const sdpa_b200_params& p) {
  const DsPlan plan = use_ds_backward(p) ? ds_plan(p) : DsPlan();
  const size_t with_ds = plan.tiles > 0 ? bwd_vector_bytes(p) + ds_workspace_bytes(p, plan) : 0;
  const size_t least = bwd_workspace_min_bytes(p);
  return with_ds > least ? with_ds : least;
}

int launch_bwd(const sdpa_b200_params& p, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  const bool f16 = p.dtype == SDPA_B200_F16;
  const bool varlen = p.cu_seqlens_q != nullptr;
  const int lq_pad = lq_padded(p);
  const size_t vec_elems = static_cast<size_t>(p.batch) * p.heads_q * lq_pad;
  float* nlse2 = reinterpret_cast<float*>(static_cast<char*>(workspace) + kWorkspaceHeaderBytes);
  float* ndelta = nlse2 + vec_elems;

  PreParams pre;
  pre.out = static_cast<const uint16_t*>(p.out);
  pre.dout = static_cast<const uint16_t*>(p.dout);
  pre.lse = p.lse;
  pre.nlse2 = nlse2;
  pre.ndelta = ndelta;
  pre.cu_q = p.cu_seqlens_q;
  pre.o_batch_stride = p.o_batch_stride;
  pre.o_head_stride = p.o_head_stride;
  pre.o_row_stride = p.o_row_stride;
  pre.do_batch_stride = p.do_batch_stride;
  pre.do_head_stride = p.do_head_stride;
  pre.do_row_stride = p.do_row_stride;
  pre.seqlen_q = p.max_seqlen_q;
  pre.total_q = p.total_q;
  pre.heads_q = p.heads_q;
  pre.lq_pad = lq_pad;
  pre.head_dim = p.head_dim;
  pre.grads = packed_grads(p);
  const bool fused = use_fused_backward(p);
  const DsPlan plan = use_ds_backward(p) ? ds_plan(p) : DsPlan();
  const bool through_ds = plan.tiles > 0 && workspace_bytes >= kWorkspaceHeaderBytes + bwd_workspace_bytes(p);
  char* behind_vectors = static_cast<char*>(workspace) + kWorkspaceHeaderBytes + bwd_vector_bytes(p);
  pre.ds_seq_base = through_ds && varlen ? reinterpret_cast<int32_t*>(behind_vectors) : nullptr;
  pre.cu_k = p.cu_seqlens_k;
  pre.is_causal = p.is_causal;
  float* dq_acc = fused ? reinterpret_cast<float*>(static_cast<char*>(workspace) + kWorkspaceHeaderBytes + bwd_vector_bytes(p)) : nullptr;
  pre.dq_acc = dq_acc;
  pre.dq_acc_rows = fused && varlen ? static_cast<int>(bwd_fused_acc_rows(p, lq_pad) / p.heads_q) : 0;
  auto pick_pre = [&](auto dim_tag) {
    constexpr int kD = decltype(dim_tag)::value;
    return varlen ? (f16 ? bwd_preprocess_kernel<kD, true, true> : bwd_preprocess_kernel<kD, false, true>)
                  : (f16 ? bwd_preprocess_kernel<kD, true, false> : bwd_preprocess_kernel<kD, false, false>);
  };
  auto pre_kernel = p.head_dim <= 64 ? pick_pre(std::integral_constant<int, 64>{}) : pick_pre(std::integral_constant<int, 128>{});
  const int pre_rows = p.head_dim <= 64 ? kPreRows<64> : kPreRows<128>;
  int pre_blocks = lq_pad / pre_rows;
  if (varlen) {
    // The mean length's, but a third of the longest one's, since a block that goes on pays one memory latency each time, and no fewer than the SMs hold at once: below
    // that a latency is all there is (all rows' blocks at once | by the mean and the third | so, us: 4 of 64 to 2048, 2 heads, D128 3.5 | 4.4 | 3.5, 1024 + 64, one head 2.7 | 3.3 | 2.9,
    // 3000 + 100, 8 heads, D64 3.4 | 3.9 | 3.3, one of 2048 among 3 of 16, 8 heads, D128 6.1 | 5.7 | 5.4).
    const int64_t mean = p.total_q / p.batch / pre_rows + 1, third = (pre_blocks + 2) / 3;
    const int64_t held = kPreBlocks<true> * kSms / (static_cast<int64_t>(p.heads_q) * p.batch);
    pre_blocks = static_cast<int>(std::min<int64_t>({std::max({mean, third, held}), pre_blocks, kMaxGridY}));
  }
  for (pre.block0 = 0; pre.block0 < pre_blocks; pre.block0 += kMaxGridY) {  // one launch up to 2 M rows
    const int rest = pre_blocks - pre.block0;
    const dim3 pre_grid(p.heads_q + (varlen ? 1 : 0), rest < kMaxGridY ? rest : kMaxGridY, p.batch);
    pre_kernel<<<pre_grid, 256, 0, stream>>>(pre);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
      set_error("backward preprocess: launch failed: %s", cudaGetErrorString(err));
      return SDPA_B200_LAUNCH_FAILED;
    }
    count_launch();
  }

  CUtensorMap tm_q, tm_k, tm_v, tm_do;
  const int64_t rows_q = varlen ? p.total_q : p.max_seqlen_q;
  const int64_t rows_k = varlen ? p.total_k : p.max_seqlen_k;
  const int64_t nb = varlen ? 1 : p.batch;
  int st;
  const int box = p.head_dim <= 64 && !fused ? 64 : kTile;  // rows; tiles of 128 take two
  if ((st = make_tensor_map_16(f16, &tm_q, p.q, p.head_dim, rows_q, p.heads_q, nb, p.q_row_stride, p.q_head_stride,
                                 p.q_batch_stride, box)) != SDPA_B200_OK)
    return st;
  if ((st = make_tensor_map_16(f16, &tm_k, p.k, p.head_dim, rows_k, p.heads_kv, nb, p.k_row_stride, p.k_head_stride,
                                 p.k_batch_stride, box)) != SDPA_B200_OK)
    return st;
  if ((st = make_tensor_map_16(f16, &tm_v, p.v, p.head_dim, rows_k, p.heads_kv, nb, p.v_row_stride, p.v_head_stride,
                                 p.v_batch_stride, box)) != SDPA_B200_OK)
    return st;
  if ((st = make_tensor_map_16(f16, &tm_do, p.dout, p.head_dim, rows_q, p.heads_q, nb, p.do_row_stride,
                                 p.do_head_stride, p.do_batch_stride, box)) != SDPA_B200_OK)
    return st;
  CUtensorMap tm_dk, tm_dv;  // outputs, stored tile by tile from the epilogue's staging buffers
  if ((st = make_tensor_map_16(f16, &tm_dk, p.dk, p.head_dim, rows_k, p.heads_kv, nb, p.dk_row_stride, p.dk_head_stride,
                                 p.dk_batch_stride, kTile)) != SDPA_B200_OK)
    return st;
  if ((st = make_tensor_map_16(f16, &tm_dv, p.dv, p.head_dim, rows_k, p.heads_kv, nb, p.dv_row_stride, p.dv_head_stride,
                                 p.dv_batch_stride, kTile)) != SDPA_B200_OK)
    return st;

  BwdKernelParams kp;
  kp.nlse2 = nlse2;
  kp.ndelta = ndelta;
  kp.dq = static_cast<uint16_t*>(p.dq);
  kp.dk = static_cast<uint16_t*>(p.dk);
  kp.dv = static_cast<uint16_t*>(p.dv);
  kp.cu_q = p.cu_seqlens_q;
  kp.cu_k = p.cu_seqlens_k;
  kp.status = p.device_status != nullptr ? p.device_status : static_cast<uint32_t*>(workspace);
  kp.dq_batch_stride = p.dq_batch_stride;
  kp.dq_head_stride = p.dq_head_stride;
  kp.dq_row_stride = p.dq_row_stride;
  kp.dk_batch_stride = p.dk_batch_stride;
  kp.dk_head_stride = p.dk_head_stride;
  kp.dk_row_stride = p.dk_row_stride;
  kp.dv_batch_stride = p.dv_batch_stride;
  kp.dv_head_stride = p.dv_head_stride;
  kp.dv_row_stride = p.dv_row_stride;
  kp.seqlen_q = p.max_seqlen_q;
  kp.seqlen_k = p.max_seqlen_k;
  kp.heads_q = p.heads_q;
  kp.heads_kv = p.heads_kv;
  kp.kv_group = p.heads_q / p.heads_kv;
  kp.lq_pad = lq_pad;
  kp.scale = p.softmax_scale;
  kp.head_dim = p.head_dim;
  const bool drop = p.dropout_p > 0.f;
  kp.keep_rows = drop ? p.keep_rows : nullptr;
  kp.keep_cols = drop ? p.keep_cols : nullptr;
  kp.keep_lq_pad = (p.max_seqlen_q + 127) / 128 * 128;
  kp.keep_lk_pad = (p.max_seqlen_k + 127) / 128 * 128;
  kp.keep_q_rows = p.cu_seqlens_q != nullptr ? p.total_q + 128 : kp.keep_lq_pad;
  kp.keep_k_rows = p.cu_seqlens_q != nullptr ? p.total_k + 128 : kp.keep_lk_pad;
  kp.keep_scale = drop ? 1.f / (1.f - p.dropout_p) : 1.f;
  kp.bias = static_cast<const uint16_t*>(p.bias);
  kp.bias_batch_stride = p.bias_batch_stride;
  kp.bias_head_stride = p.bias_head_stride;
  kp.bias_row_stride = p.bias_row_stride;
  kp.bias_t = static_cast<const uint16_t*>(p.bias_t);
  kp.bias_t_batch_stride = p.bias_t_batch_stride;
  kp.bias_t_head_stride = p.bias_t_head_stride;
  kp.bias_t_row_stride = p.bias_t_row_stride;
  kp.dbias = static_cast<uint16_t*>(p.dbias);
  kp.dbias_batch_stride = p.dbias_batch_stride;
  kp.dbias_head_stride = p.dbias_head_stride;
  kp.dbias_row_stride = p.dbias_row_stride;
  kp.inv_scale = 1.f / p.softmax_scale;
  kp.scale_log2 = p.softmax_scale * 1.4426950408889634f;
  kp.is_causal = p.is_causal;
#ifdef SDPA_BWD_STAMPS
  {
    const char* env = getenv("SDPA_BWD_STAMPS_PTR");
    kp.stamps = env ? reinterpret_cast<float*>(strtoull(env, nullptr, 10)) : nullptr;
  }
#endif

  // streamed: q + dO of the group, or k + v
  // `rows`: what the stationary blocks divide; a head streams `rows_streamed` rows of `streams` heads
  auto set_order = [&](int heads_x, int rows, int heads, int rows_streamed, int streams, double packed_rows) {
    kp.heads_x = heads_x;
    const double row_bytes = 2.0 * p.head_dim * 2;
    kp.order = block_order(heads, (rows + kTile - 1) / kTile,
                           varlen && !fused && p.is_causal ? heads_per_packed_group(row_bytes * packed_rows, heads)
                                                           : heads_per_l2_group(row_bytes * rows_streamed * streams, heads, 48.0 * 1024 * 1024, !fused && !varlen));
    return kp.order.slots;
  };
  const double rows_q_all = static_cast<double>(p.total_q) * p.heads_q, rows_k_all = static_cast<double>(p.total_k) * p.heads_kv;
  kp.bh0 = 0;
  kp.split = bwd_split(p);
  kp.ds.data = nullptr;
  kp.ds_call = plan.tiles > 0;
  if (through_ds) {
    kp.ds.data = reinterpret_cast<uint16_t*>(behind_vectors + ds_table_bytes(p));
    kp.ds.seq_base = pre.ds_seq_base;
    kp.ds.capacity = plan.tiles;
    kp.ds_counter = static_cast<uint32_t*>(workspace) + 2;
    const int kv_heads = p.batch * p.heads_kv;
    for (int first = 0; first < kv_heads; first += plan.kv_heads) {
      const int n = kv_heads - first < plan.kv_heads ? kv_heads - first : plan.kv_heads;
      kp.bh0 = first;
      kp.ds.head0 = first * kp.kv_group;
      const int grid = set_order(p.heads_kv, p.max_seqlen_k, n, p.max_seqlen_q, kp.kv_group, rows_q_all);
      if ((st = launch_tile_kernel(kModeDKDV, p.head_dim, f16, grid, true, stream, tm_q, tm_k, tm_v, tm_do, tm_dv, tm_dk, kp,
                                   /*overlap_previous=*/first == 0)) != SDPA_B200_OK)
        return st;
      if ((st = launch_bwd_ds_gemm(p, kp.ds, first, n, false, kp.ds_counter, kp.status, stream)) != SDPA_B200_OK) return st;
    }
    return SDPA_B200_OK;
  }
  const int grid_dkdv = set_order(p.heads_kv, p.max_seqlen_k, p.batch * p.heads_kv, p.max_seqlen_q, kp.kv_group, rows_q_all);
  if (fused) return launch_bwd_fused(p, kp, dq_acc, grid_dkdv, stream, tm_q, tm_k, tm_v, tm_do, tm_dv, tm_dk);
  CUtensorMap tm_dq;
  if ((st = make_tensor_map_16(f16, &tm_dq, p.dq, p.head_dim, rows_q, p.heads_q, nb, p.dq_row_stride, p.dq_head_stride,
                                 p.dq_batch_stride, kTile)) != SDPA_B200_OK)
    return st;
  // a packed call's blocks are those with rows: half a block more per sequence and head than the rows fill
  const auto blocks = [&](int grid, int heads, int rows) { return varlen ? heads * (rows / static_cast<double>(kTile) + 0.5 * p.batch) : grid; };
  const auto tiles = [](int rows) { return (rows + kTile - 1) / kTile; };
  const bool wide_dkdv = wide_tiles(blocks(grid_dkdv, p.heads_kv, p.total_k), kp.kv_group * tiles(p.max_seqlen_q));
  BwdKernelParams kq = kp;
  std::swap(kp, kq);
  const int grid_dq = set_order(p.heads_q, p.max_seqlen_q, p.batch * p.heads_q, p.max_seqlen_k, 1, rows_k_all);
  std::swap(kp, kq);  // kp: the dK/dV kernel's, kq: the dQ kernel's
  const bool wide_dq = wide_tiles(blocks(grid_dq, p.heads_q, p.total_q), tiles(p.max_seqlen_k));
  // Both in one launch where the same instance serves both, with the dQ blocks behind the dK/dV blocks as the overlapped launches have them: about 2.5 us less of
  // host time, which is what bounds the steps of short sequences, and no gap (step, two launches | one, us: B4 H8 L500 D64 f16 83.3 | 78.2, B1 H8 L2048 D128
  // 74.1 | 71.5, B16 H16 L500 D64 120.8 | 116.6, B8 H12 L1000 D64 unmasked 187 | 181, B32 H12 L300 D64 with dropout 173.8 | 168.5; backward alone, replayed from a graph: B8 H12 L512
  // D64 with a mask 50.4 | 48.1, B1 H8 L2048 D128 34.9 | 33.3, B4 H8 L512 D128 24.1 | 24.1). Above head_dim 64 two launches where all blocks fit the SMs at once, although one
  // is shorter there too (step B1 H16 L512 D128 83.9 | 82.4, B4 H8 L256 D96 83.5 | 80.5; backward alone from a graph 14.9 | 14.2, 11.7 | 11.0): a test counts them.
  const bool pair = !kp.ds_call && kp.split == 1 && (p.head_dim > 64 || wide_dkdv == wide_dq) && (kp.bias == nullptr || (kp.bias_row_stride == 0 && kp.dbias == nullptr)) &&
                    (p.head_dim <= 64 || grid_dkdv + grid_dq > kSms);
  if (pair)
    return launch_tile_pair(p.head_dim, f16, grid_dkdv, grid_dq, DqGrid{kq.order, kq.heads_x, grid_dkdv}, wide_dkdv, stream, tm_q, tm_k, tm_v, tm_do, tm_dv, tm_dk, tm_dq, kp);
  if ((st = launch_tile_kernel(kModeDKDV, p.head_dim, f16, grid_dkdv, wide_dkdv, stream, tm_q, tm_k, tm_v, tm_do, tm_dv, tm_dk, kp,
                               /*overlap_previous=*/true)) != SDPA_B200_OK)
    return st;
  return launch_tile_kernel(kModeDQ, p.head_dim, f16, grid_dq, wide_dq, stream, tm_q, tm_k, tm_v, tm_do, tm_dq, tm_dq, kq,
                            /*overlap_previous=*/true);
}

}  // namespace sdpa_b200
