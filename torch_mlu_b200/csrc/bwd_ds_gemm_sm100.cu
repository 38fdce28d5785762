// dQ = scale dS K (and, for head dims above 128, dK = scale dS^T Q) from the dS tiles that the key-block kernel of the backward
// has left in the workspace (ds_tiles.cuh).
//
// Bound by memory: every dS tile is read once, 32 KB for 128 x 128 x head_dim multiply-adds. Two 128-row tiles per unit share each B
// block (48 KB per step of 64 at head_dim 128 where single tiles would read 64). B8 H16 L2048 D128 causal: 0.57 GB of dS in 122 us. What the kernel in front
// wrote last is read first, from L2, which is asked to give dS up when it has been read (up to head_dim 128, where it is read once): 130 us -> 122 there, packed 12 of 64 to
// 2048 tokens, 16/4 heads, 78 -> 72. Above, where dK and dQ read it and L2 keeps it for neither, the hint changed nothing. Stores of dS that ask L2 to keep it save
// 3 us more here (119), but neither the read nor its hint takes that back: the lines stay in L2 when the call is over, and every kernel behind has less of it
// (the pre-pass of B8 H16 L2048 21.5 -> 22.7 us; an addition over 48 + 48 MB, repeated, 12.5 -> 13.7; a product of two 4096 x 4096 matrices 88.9 -> 90.1).
//
// Persistent: one CTA per SM takes units of 256 output rows (two 128-row tiles that share every B block) of one head from a
// counter, heaviest first inside a group of heads. Per 64 rows of the contraction a stage brings B (64 rows of K or Q, 128-byte
// swizzle) and the two tiles' 128 x 64 slices of dS (16 KB each, no swizzle: the image in the workspace is the operand). Warp 8
// claims units and loads, warp 9 issues the MMAs, warps 0-7 (thread = output row) scale, convert and store.
#include <cuda_bf16.h>

#include "bwd_ds_gemm.h"
#include "ptx_sm100.cuh"

namespace sdpa_b200 {
namespace {

constexpr int kThreads = 320;
constexpr int kStep = 64;                       // contraction rows per stage
constexpr int kPair = 2 * kDsTile;              // output rows per unit
constexpr uint32_t kBoxBytes = kStep * 128;     // 64 rows x 64 columns
constexpr uint32_t kSliceBytes = kDsTile * kStep * 2;
__host__ __device__ constexpr uint32_t stage_bytes(int d) { return d / 64 * kBoxBytes + 2 * kSliceBytes; }
__host__ __device__ constexpr int stages_for(int d) { return d == 256 ? 3 : 4; }
__host__ __device__ constexpr uint32_t stage_out_off(int d) { return stages_for(d) * stage_bytes(d); }  // 4 KB per warp
__host__ __device__ constexpr uint32_t bars_off(int d) { return stage_out_off(d) + 8 * 4096; }

constexpr uint32_t kBarFull = 0;                   // stages
constexpr uint32_t kBarEmpty = kBarFull + 8 * 4;   // stages
constexpr uint32_t kBarUnitFull = kBarEmpty + 8 * 4;   // 2
constexpr uint32_t kBarUnitEmpty = kBarUnitFull + 16;  // 2, 8 warps
constexpr uint32_t kBarAccFull = kBarUnitEmpty + 16;   // 2
constexpr uint32_t kBarAccFree = kBarAccFull + 16;     // 2, 8 warps
constexpr uint32_t kFlags = kBarAccFree + 16;          // one word per stage
constexpr uint32_t kUnits = kFlags + 16;               // 2 x 32 bytes
constexpr uint32_t kTmemPtr = kUnits + 64;
constexpr uint32_t kAbort = kTmemPtr + 4;
__host__ __device__ constexpr uint32_t smem_bytes(int d) { return bars_off(d) + 512 + 1024; }
static_assert(kAbort + 4 <= 512 && smem_bytes(128) <= 232448 && smem_bytes(256) <= 232448,
              "shared memory map does not fit");

constexpr uint32_t kFlagTile0 = 1, kFlagTile1 = 2, kFlagFirst = 4, kFlagLast = 8, kFlagStop = 16, kFlagKeys = 32;
constexpr int kUnitStop = 2;

// A unit in the table is two int4:
//   kind (0 dQ, 1 dK, kUnitStop), first output row within the sequence, output rows of the sequence, its first row in a packed tensor
//   head, batch, bit t: some contraction row contributes to tile t, unused

// D[tmem] (+)= A[smem, no swizzle] * B[smem, 128-byte swizzle]
__device__ __forceinline__ void umma_ss_plain_a(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t"
      "}\n" ::"r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(kDescHiSw128), "r"(idesc), "r"(accumulate)
      : "memory");
}

// One stage of one tile: ACC (128 x n) (+)= slice * B. Without swizzle an operand is made of 8 x 16-byte core matrices of 128
// contiguous bytes. dQ (kKeys false): the slice is [16 query groups][64 keys][8 queries], MN-major: query groups are 1024 bytes
// apart (SBO), groups of 8 keys 128 (LBO), a step of 16 keys 256. dK: [8 query groups][128 keys][8 queries], K-major: groups of
// 8 keys 128 bytes apart (SBO), query groups 2048 (LBO), a step of 16 queries 4096.
template <bool kKeys>
__device__ __forceinline__ void issue_stage(uint32_t acc, uint32_t slice, uint32_t b_smem, uint32_t idesc, bool accumulate) {
  constexpr uint32_t kLbo = kKeys ? 2048 : 128, kSbo = kKeys ? 128 : 1024, kAdvance = kKeys ? 4096 : 256;
  const uint32_t a_lo = (slice >> 4) | ((kLbo >> 4) << 16);
  const uint32_t a_hi = (kSbo >> 4) | (1u << 14);
  const uint32_t b_lo = umma_desc_lo_mnmajor(b_smem, kBoxBytes);
#pragma unroll
  for (int ks = 0; ks < kStep / 16; ++ks)
    umma_ss_plain_a(acc, a_lo + ks * (kAdvance >> 4), a_hi, b_lo + ks * (2048 >> 4), idesc, (accumulate || ks > 0) ? 1u : 0u);
}

template <int kD, bool kF16>
__global__ void __launch_bounds__(kThreads, 1)
bwd_ds_gemm_kernel(const __grid_constant__ CUtensorMap tm_ds_q, const __grid_constant__ CUtensorMap tm_ds_k,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_q,
                   const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dk, const DsGemmParams p) {
  constexpr int kStages = stages_for(kD);
  constexpr uint32_t kStageBytes = stage_bytes(kD);
  constexpr int kAccs = kD == 256 ? 1 : 2;  // accumulator pairs in tensor memory
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t bar = base + bars_off(kD);
  uint8_t* bar_ptr = smem + bars_off(kD);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(bar_ptr + kAbort);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(bar_ptr + kTmemPtr);
  volatile uint32_t* flags = reinterpret_cast<volatile uint32_t*>(bar_ptr + kFlags);
  int4* units = reinterpret_cast<int4*>(bar_ptr + kUnits);

  if (warp == 8 && lane == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar + kBarFull + 8 * s, 1);
      mbar_init(bar + kBarEmpty + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar + kBarUnitFull + 8 * i, 1);
      mbar_init(bar + kBarUnitEmpty + 8 * i, 8);
      mbar_init(bar + kBarAccFull + 8 * i, 1);
      mbar_init(bar + kBarAccFree + 8 * i, 8);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_ds_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_dq);
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(bar + kTmemPtr, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp == 8) {
    // ------------------------------------------------------------------ unit claims and TMA loads
    if (elect_one()) {
      // everything above runs under the tail of the grid that writes dS and clears the counter
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const uint32_t boxes = (p.head_dim + 63) / 64;
      const uint64_t read_once = l2_drop();
      uint32_t stage = 0, unit_count = 0;
      bool ok = true;
      uint32_t u = atomicAdd(p.counter, 1u);
      while (ok && u < p.units) {
        const uint32_t next = atomicAdd(p.counter, 1u);  // in flight under this unit's loads
        // unit -> (group of KV heads, dK or dQ, rank in the group, head)
        int grp = static_cast<int>(u / p.units_per_group);
        int w = static_cast<int>(u - grp * p.units_per_group);
        grp = p.num_groups - 1 - grp;  // the dS written last is still in L2
        const int kv_heads = min(p.heads_per_group, p.num_kv_heads - grp * p.heads_per_group);
        const bool keys = w < p.key_units_per_group;
        if (!keys) w -= p.key_units_per_group;
        const int size = keys ? kv_heads : kv_heads * p.kv_group;
        const int rank = w / size, pairs = keys ? p.key_pairs : p.query_pairs;
        if (rank < pairs) {  // else: padding of a short last group
          const int hx = w - rank * size;  // head within the group
          const int kvh = p.kv_head0 + grp * p.heads_per_group + (keys ? hx : hx / p.kv_group);  // batch * heads_kv + head
          const int b = kvh / p.heads_kv;
          const int hkv = kvh - b * p.heads_kv;
          const int hq = keys ? hkv * p.kv_group : hkv * p.kv_group + hx % p.kv_group;
          int q_off = 0, k_off = 0, len_q = p.seqlen_q, len_k = p.seqlen_k, bcoord = b;
          if (p.cu_q != nullptr) {
            q_off = p.cu_q[b];
            len_q = p.cu_q[b + 1] - q_off;
            k_off = p.cu_k[b];
            len_k = p.cu_k[b + 1] - k_off;
            bcoord = 0;
          }
          const int off = len_k - len_q;
          // heaviest first: key pair 0 (of a packed sequence: by the pairs behind it), the last query pair
          const int rows = keys ? len_k : len_q;
          const int pair = keys ? rank - (pairs - (len_k + kPair - 1) / kPair) : pairs - 1 - rank;
          const int row0 = pair * kPair;
          if (row0 >= 0 && row0 < rows) {
            // steps [lo, hi) of 64 contraction rows that contribute to tile t
            int lo[2] = {0, 0}, hi[2] = {0, 0};
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              const int x0 = row0 + t * kDsTile;
              if (x0 >= rows) continue;
              if (keys) {
                hi[t] = (len_q + kStep - 1) / kStep;
                if (p.is_causal) {
                  lo[t] = max(0, (x0 - off) / kStep);
                  if (x0 - off > len_q - 1) lo[t] = hi[t];
                }
              } else {
                const int end = p.is_causal ? min(len_k, x0 + kDsTile + off) : len_k;
                hi[t] = end > 0 ? (end + kStep - 1) / kStep : 0;
              }
              if (hi[t] < lo[t]) hi[t] = lo[t];
            }
            const bool has0 = hi[0] > lo[0], has1 = hi[1] > lo[1];
            const int first = has0 ? (has1 ? min(lo[0], lo[1]) : lo[0]) : lo[1];
            const int last = has0 ? (has1 ? max(hi[0], hi[1]) : hi[0]) : hi[1];
            const int slot = unit_count & 1;
            ok = mbar_wait(bar + kBarUnitEmpty + 8 * slot, ((unit_count >> 1) & 1) ^ 1, abort_flag);
            if (!ok) break;
            units[2 * slot] = make_int4(keys ? 1 : 0, row0, rows, keys ? k_off : q_off);
            units[2 * slot + 1] = make_int4(keys ? hkv : hq, b, (has0 ? 1 : 0) | (has1 ? 2 : 0), 0);
            mbar_arrive(bar + kBarUnitFull + 8 * slot);
            ++unit_count;
            const int n_heads = keys ? p.kv_group : 1;
            for (int hi_q = 0; ok && hi_q < n_heads; ++hi_q) {
              const DsHead ds = ds_head(p.ds, b, hq + hi_q, p.heads_q, len_q, len_k, p.is_causal != 0);
              for (int ks = first; ks < last; ++ks, ++stage) {
                const int s = stage % kStages;
                ok = mbar_wait(bar + kBarEmpty + 8 * s, ((stage / kStages) & 1) ^ 1, abort_flag);
                if (!ok) break;
                const bool on0 = ks >= lo[0] && ks < hi[0], on1 = ks >= lo[1] && ks < hi[1];
                const uint32_t full = bar + kBarFull + 8 * s, dst = base + s * kStageBytes;
                flags[s] = (on0 ? kFlagTile0 : 0u) | (on1 ? kFlagTile1 : 0u) | (keys ? kFlagKeys : 0u) |
                           (hi_q == 0 && ks == first ? kFlagFirst : 0u) |
                           (hi_q == n_heads - 1 && ks == last - 1 ? kFlagLast : 0u);
                mbar_arrive_expect_tx(full, boxes * kBoxBytes + (on0 ? kSliceBytes : 0u) + (on1 ? kSliceBytes : 0u));
                const CUtensorMap* tm_b = keys ? &tm_q : &tm_k;
                const int b_row = (keys ? q_off : k_off) + ks * kStep, b_head = keys ? hq + hi_q : hkv;
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                  if (!(t == 0 ? on0 : on1)) continue;
                  const int x = row0 / kDsTile + t;  // tile of output rows
                  const uint32_t a_dst = dst + kD / 64 * kBoxBytes + t * kSliceBytes;
                  if (keys) {
                    const int tile = static_cast<int>(ds.tile(ks >> 1, x));
                    tma_load_4d(a_dst, &tm_ds_k, full, 0, tile * 16 + (ks & 1) * 8, 0, 0);
                  } else {
                    const int tile = static_cast<int>(ds.tile(x, ks >> 1));
                    if constexpr (kD == 128) tma_load_4d_hint(a_dst, &tm_ds_q, full, (ks & 1) * 128, tile * 16, 0, 0, read_once);
                    else tma_load_4d(a_dst, &tm_ds_q, full, (ks & 1) * 128, tile * 16, 0, 0);
                  }
                }
                for (uint32_t c = 0; c < boxes; ++c) tma_load_4d(dst + c * kBoxBytes, tm_b, full, c * 64, b_row, b_head, bcoord);
              }
            }
          }
        }
        u = next;
      }
      // stop: a unit for the storing warps, an empty stage for the issuer
      if (ok) {
        const int slot = unit_count & 1;
        ok = mbar_wait(bar + kBarUnitEmpty + 8 * slot, ((unit_count >> 1) & 1) ^ 1, abort_flag);
        if (ok) {
          units[2 * slot] = make_int4(kUnitStop, 0, 0, 0);
          mbar_arrive(bar + kBarUnitFull + 8 * slot);
          const int s = stage % kStages;
          ok = mbar_wait(bar + kBarEmpty + 8 * s, ((stage / kStages) & 1) ^ 1, abort_flag);
          if (ok) {
            flags[s] = kFlagStop;
            mbar_arrive(bar + kBarFull + 8 * s);
          }
        }
      }
      drain_after_abort(abort_flag);
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t n = (p.head_dim + 15) / 16 * 16;  // columns that exist; M = 128 takes any multiple of 16
      const uint32_t idesc_q = umma_idesc_16(kDsTile, 16, true, true, kF16) + ((n - 16) << 14);
      const uint32_t idesc_k = umma_idesc_16(kDsTile, 16, false, true, kF16) + ((n - 16) << 14);
      uint32_t acc_count = 0;
      bool started0 = false, started1 = false;
      for (uint32_t stage = 0;; ++stage) {
        const int s = stage % kStages;
        if (!mbar_wait(bar + kBarFull + 8 * s, (stage / kStages) & 1, abort_flag)) break;
        const uint32_t f = flags[s];
        if (f & kFlagStop) break;
        const uint32_t a = acc_count % kAccs;
        if (f & kFlagFirst) {
          if (!mbar_wait(bar + kBarAccFree + 8 * a, ((acc_count / kAccs) & 1) ^ 1, abort_flag)) break;
          started0 = started1 = false;
        }
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + a * (2 * kD);
        const uint32_t b_smem = base + s * kStageBytes, slices = b_smem + kD / 64 * kBoxBytes;
        if (f & kFlagTile0) {
          if (f & kFlagKeys) issue_stage<true>(acc, slices, b_smem, idesc_k, started0);
          else issue_stage<false>(acc, slices, b_smem, idesc_q, started0);
          started0 = true;
        }
        if (f & kFlagTile1) {
          if (f & kFlagKeys) issue_stage<true>(acc + kD, slices + kSliceBytes, b_smem, idesc_k, started1);
          else issue_stage<false>(acc + kD, slices + kSliceBytes, b_smem, idesc_q, started1);
          started1 = true;
        }
        umma_commit(bar + kBarEmpty + 8 * s);
        if (f & kFlagLast) {
          umma_commit(bar + kBarAccFull + 8 * a);
          ++acc_count;
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ scale, convert, store (thread = output row)
    const int t = warp >> 2;
    const int r_warp = t * kDsTile + (warp & 3) * 32;  // first row of this warp in the unit
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t staging = base + stage_out_off(kD) + warp * 4096;
    uint8_t* staging_row = smem + stage_out_off(kD) + warp * 4096 + lane * 128;
    uint32_t acc_count = 0;
    for (uint32_t i = 0;; ++i) {
      const int slot = i & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(bar + kBarUnitFull + 8 * slot, (i >> 1) & 1, abort_flag))) break;
      const int4 u0 = units[2 * slot], u1 = units[2 * slot + 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(bar + kBarUnitEmpty + 8 * slot);
      if (u0.x == kUnitStop) break;
      const int row = u0.y + r_warp;      // this warp's first row within the sequence
      const int rows = u0.z - row;        // rows of it that exist (may be negative)
      const bool any = u1.z != 0, mine = ((u1.z >> t) & 1) != 0;
      const uint32_t a = acc_count % kAccs;
      if (any) {
        if (!__all_sync(0xffffffffu, mbar_wait(bar + kBarAccFull + 8 * a, (acc_count / kAccs) & 1, abort_flag))) break;
        ++acc_count;
        tc_fence_after_sync();
      }
      const bool keys = u0.x != 0;
      const bool packed = p.cu_q != nullptr;
      // a packed tile that ends inside its sequence's last rows would spill into the next sequence: row by row then
      const bool use_tma = !packed || rows >= 32;
      uint16_t* orow = nullptr;
      if (!use_tma) {
        const int64_t orow_index = u0.w + row + lane;
        orow = keys ? p.dk + orow_index * p.dk_row_stride + u1.x * p.dk_head_stride
                    : p.dq + orow_index * p.dq_row_stride + u1.x * p.dq_head_stride;
      }
      const CUtensorMap* tm = keys ? &tm_dk : &tm_dq;
#pragma unroll
      for (int c = 0; c < kD / 64; ++c) {
        uint32_t v[64];
        if (mine) {
          tmem_ld_x64(tmem_base + a * (2 * kD) + t * kD + c * 64 + lane_base, v);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < 64; ++j) v[j] = 0u;
        }
        if (any && c == kD / 64 - 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar + kBarAccFree + 8 * a);
        }
        if (rows <= 0 || c * 64 >= p.head_dim) continue;
        uint4 w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          w[j].x = pack_16x2<kF16>(__uint_as_float(v[8 * j + 0]) * p.scale, __uint_as_float(v[8 * j + 1]) * p.scale);
          w[j].y = pack_16x2<kF16>(__uint_as_float(v[8 * j + 2]) * p.scale, __uint_as_float(v[8 * j + 3]) * p.scale);
          w[j].z = pack_16x2<kF16>(__uint_as_float(v[8 * j + 4]) * p.scale, __uint_as_float(v[8 * j + 5]) * p.scale);
          w[j].w = pack_16x2<kF16>(__uint_as_float(v[8 * j + 6]) * p.scale, __uint_as_float(v[8 * j + 7]) * p.scale);
        }
        if (use_tma) {
          if (lane == 0) tma_store_wait_read();  // the previous 64 columns have left the staging rows
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(staging_row + ((j ^ (lane & 7)) << 4)) = w[j];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_4d(tm, staging, c * 64, u0.w + row, u1.x, packed ? 0 : u1.y);
            tma_store_commit();
          }
        } else if (lane < rows) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (c * 64 + j * 8 < p.head_dim) *reinterpret_cast<uint4*>(orow + c * 64 + j * 8) = w[j];
        }
      }
    }
    if (lane == 0) tma_store_wait_read();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag != 0) atomicExch(p.status, static_cast<uint32_t>(SDPA_B200_DEVICE_TIMEOUT));
}

using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                        const CUtensorMap, const DsGemmParams);

Kernel pick_kernel(int head_dim, bool f16) {
  if (head_dim <= 128) return f16 ? bwd_ds_gemm_kernel<128, true> : bwd_ds_gemm_kernel<128, false>;
  return f16 ? bwd_ds_gemm_kernel<256, true> : bwd_ds_gemm_kernel<256, false>;
}

}  // namespace

// dS of a call (half of B H Lq Lk elements of two bytes under a causal mask) may take this much of the workspace; a dense call with
// more of it goes through it in several passes over its KV heads. One pass is best (step of B8 H16 L2048, 0.57 GB of dS: 673 us in
// one pass, 709 in two, 766 in six, where a pass's dS would stay in L2; B2 H16 L8192, 2.18 GB: 2189 in its two passes, 2115 in one
// with room for it).
constexpr size_t kDsBytesMax = size_t{2} << 30;

DsPlan ds_plan(const sdpa_b200_params& p) {
  DsPlan plan;
  const int64_t cap = static_cast<int64_t>(kDsBytesMax / kDsTileBytes);
  const int64_t key_tiles = (static_cast<int64_t>(p.max_seqlen_k) + kDsTile - 1) / kDsTile;
  const int64_t kv_heads = static_cast<int64_t>(p.batch) * p.heads_kv;
  if (p.cu_seqlens_q != nullptr) {
    // the lengths are on the device: every query tile there can be, against the longest keys
    const int64_t tiles = (p.total_q / kDsTile + p.batch) * key_tiles * p.heads_q;
    if (tiles > cap) return plan;
    plan.kv_heads = static_cast<int>(kv_heads);
    plan.tiles = static_cast<uint32_t>(tiles);
    return plan;
  }
  const int64_t per_kv_head = p.heads_q / p.heads_kv * ds_tiles_per_head(p.max_seqlen_q, p.max_seqlen_k, p.is_causal != 0);
  if (per_kv_head <= 0 || per_kv_head > cap) return plan;
  const int64_t passes = (kv_heads * per_kv_head + cap - 1) / cap;
  int64_t per_pass = (kv_heads + passes - 1) / passes;
  if (per_pass * per_kv_head > cap) per_pass = cap / per_kv_head;
  // A pass must fill the SMs a few times over, or its launches' tails cost more than the second pass over the scores: step of B1 H32/8
  // L8192 D128 causal (two passes of 256 CTAs) 2270 us with the two kernels, 2510 so; B2 (three of 384) 4524 and 4500, B1 H32/4 unmasked (two of 128)
  // 4290 and 4195. Above head_dim 128, where the alternative are three kernels, the line lies too high (B1 H32/8 L8192 D256 causal 5283, in
  // passes 4627; B2 H16/4 unmasked 9546, 7636).
  if (passes > 1 && per_pass * key_tiles < 3 * 148) return plan;
  plan.kv_heads = static_cast<int>(per_pass);
  plan.tiles = static_cast<uint32_t>(per_pass * per_kv_head);
  return plan;
}

size_t ds_table_bytes(const sdpa_b200_params& p) {
  return p.cu_seqlens_q != nullptr ? (static_cast<size_t>(p.batch) * sizeof(int32_t) + 255) / 256 * 256 : 0;
}

size_t ds_workspace_bytes(const sdpa_b200_params& p, const DsPlan& plan) {
  return plan.tiles > 0 ? ds_table_bytes(p) + plan.tiles * kDsTileBytes : 0;
}

int launch_bwd_ds_gemm(const sdpa_b200_params& p, const DsTiles& ds, int kv_head0, int num_kv_heads, bool with_dk,
                       uint32_t* counter, uint32_t* status, cudaStream_t stream) {
  const bool f16 = p.dtype == SDPA_B200_F16;
  const bool varlen = p.cu_seqlens_q != nullptr;
  const int64_t rows_q = varlen ? p.total_q : p.max_seqlen_q;
  const int64_t rows_k = varlen ? p.total_k : p.max_seqlen_k;
  const int64_t nb = varlen ? 1 : p.batch;
  CUtensorMap ds_q, ds_k, tm_k, tm_q, tm_dq, tm_dk;
  int st;
  auto map = [&](CUtensorMap* m, const void* ptr, int64_t rows, int heads, int64_t rs, int64_t hs, int64_t bs, int box) {
    return make_tensor_map_16(f16, m, ptr, p.head_dim, rows, heads, nb, rs, hs, bs, box);
  };
  if ((st = make_ds_tensor_map(&ds_q, ds.data, ds.capacity, 128, 16)) != SDPA_B200_OK) return st;
  if ((st = map(&tm_k, p.k, rows_k, p.heads_kv, p.k_row_stride, p.k_head_stride, p.k_batch_stride, kStep)) != SDPA_B200_OK) return st;
  if ((st = map(&tm_dq, p.dq, rows_q, p.heads_q, p.dq_row_stride, p.dq_head_stride, p.dq_batch_stride, 32)) != SDPA_B200_OK) return st;
  if (with_dk) {
    if ((st = make_ds_tensor_map(&ds_k, ds.data, ds.capacity, 256, 8)) != SDPA_B200_OK) return st;
    if ((st = map(&tm_q, p.q, rows_q, p.heads_q, p.q_row_stride, p.q_head_stride, p.q_batch_stride, kStep)) != SDPA_B200_OK) return st;
    if ((st = map(&tm_dk, p.dk, rows_k, p.heads_kv, p.dk_row_stride, p.dk_head_stride, p.dk_batch_stride, 32)) != SDPA_B200_OK) return st;
  } else {  // not read; encoding a map takes the host about a microsecond
    ds_k = ds_q;
    tm_q = tm_k;
    tm_dk = tm_dq;
  }

  DsGemmParams kp;
  kp.ds = ds;
  kp.cu_q = p.cu_seqlens_q;
  kp.cu_k = p.cu_seqlens_k;
  kp.counter = counter;
  kp.status = status;
  kp.dq = static_cast<uint16_t*>(p.dq);
  kp.dk = static_cast<uint16_t*>(p.dk);
  kp.dq_row_stride = p.dq_row_stride;
  kp.dq_head_stride = p.dq_head_stride;
  kp.dk_row_stride = p.dk_row_stride;
  kp.dk_head_stride = p.dk_head_stride;
  kp.seqlen_q = p.max_seqlen_q;
  kp.seqlen_k = p.max_seqlen_k;
  kp.heads_q = p.heads_q;
  kp.heads_kv = p.heads_kv;
  kp.kv_group = p.heads_q / p.heads_kv;
  kp.head_dim = p.head_dim;
  kp.is_causal = p.is_causal;
  kp.scale = p.softmax_scale;
  kp.kv_head0 = kv_head0;
  kp.num_kv_heads = num_kv_heads;
  kp.query_pairs = (p.max_seqlen_q + kPair - 1) / kPair;
  kp.key_pairs = (p.max_seqlen_k + kPair - 1) / kPair;
  // heads per group: the rows of the B operands are re-read by every unit of their head. (With dK too, groups of 1 to 8 heads, whose
  // dS might come from L2 the second time, make no difference: B4 H16 L4096 D256 576 to 580 us.)
  const double per_head = 2.0 * p.head_dim * (p.max_seqlen_k + (with_dk ? kp.kv_group * static_cast<double>(p.max_seqlen_q) : 0.0));
  const double all = 2.0 * p.head_dim * (static_cast<double>(p.total_k) * p.heads_kv + (with_dk ? static_cast<double>(p.total_q) * p.heads_q : 0.0));
  const int hpg = varlen ? heads_per_packed_group(all, num_kv_heads) : heads_per_l2_group(per_head, num_kv_heads);
  kp.heads_per_group = hpg;
  kp.key_units_per_group = with_dk ? hpg * kp.key_pairs : 0;
  kp.units_per_group = kp.key_units_per_group + hpg * kp.kv_group * kp.query_pairs;
  kp.num_groups = (num_kv_heads + hpg - 1) / hpg;
  kp.units = static_cast<uint32_t>(kp.num_groups) * kp.units_per_group;

  Kernel kernel = pick_kernel(p.head_dim, f16);
  const uint32_t smem = p.head_dim <= 128 ? smem_bytes(128) : smem_bytes(256);
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) {
    set_error("backward dS GEMM: cudaFuncSetAttribute(%u bytes smem): %s", smem, cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  const int sms = sm_count();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sms) < kp.units ? static_cast<unsigned>(sms) : kp.units);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  err = cudaLaunchKernelEx(&cfg, kernel, ds_q, ds_k, tm_k, tm_q, tm_dq, tm_dk, kp);
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("backward dS GEMM: launch failed: %s", cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  return SDPA_B200_OK;
}

}  // namespace sdpa_b200
