// Split-KV decode attention (seqlen_q == 1) for sm_100a: the HBM-bandwidth-bound member of
// the forward path. The reference has no counterpart - its dispatcher turns Lq = 1 away from
// the fused kernel (torch_mlu/csrc/aten/operators/cnnl/transformers/sdp_utils.h:510-521) -
// so semantics follow mha_varlen_fwd (FlashAttention_internal.cpp:57-267) with one query row.
//
// A unit is one (batch, kv head, chunk of up to 16 query heads of its group): all those heads ride in the M dimension of
// mma.sync.m16n8k16, so K/V bytes are read once per group. The keys of all units, cut into tiles of 64, form one list that is
// dealt out in equal contiguous shares to a grid that fits the GPU in one wave (two CTAs per SM): every SM streams the same
// number of bytes whatever the batch, the number of heads and the length are, and the loads of a CTA run on across unit
// boundaries. Where they fit as well without, whole units or clusters of CTAs that share one and merge their parts through shared memory save the
// second launch (cluster_size). (One CTA per (unit, split) left the last wave nearly empty - 512 CTAs on 444 places ran at 4.3 TB/s - and paid
// the pipeline's fill and the merge of four warps once per split.) A unit whose tiles belong to several CTAs leaves partial
// (O, lse) rows in the workspace, at most two per CTA, and a second kernel merges them.
//
// Inside a CTA each of the four warps owns 16 keys of every tile and a ring of shared-memory stages that its own elected lane
// fills by TMA (two 16 x 64-column boxes each of K and V, 128-byte swizzle: ldmatrix reads them without bank conflicts), so
// the warps never wait for one another inside a unit. 96 KB per CTA are in flight. Measured against register-fed loads and
// fixed splits (Hq 32, Hkv 8, D 128): B 64 Lk 32768 1355 -> 1223 us (7.0 TB/s; a bare read kernel reaches 7.4), B 16 Lk 8192
// 126 -> 89 us, B 1 Lk 32768 67 -> 31 us, B 1 Lk 1000 18.5 -> 8.7 us (both kernels, back to back).
#include <cuda_bf16.h>

#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "ptx_sm100.cuh"

namespace sdpa_b200 {
namespace {

constexpr int kDecWarps = 4;
constexpr int kDecThreads = kDecWarps * 32;
constexpr int kKeysPerStep = 16;                        // keys one warp handles per tile
constexpr int kTileKeys = kDecWarps * kKeysPerStep;     // 64
constexpr int kMaxSplits = 128;
constexpr int kCtasPerSm = 2;
constexpr int kMaxCluster = 8;
constexpr uint32_t kBoxRowBytes = 128;                  // one 64-column box row
constexpr uint32_t kBoxBytes = kKeysPerStep * kBoxRowBytes;

struct DecodeParams {
  const uint16_t* q;  // bf16 or f16 bits (f16 != 0)
  uint16_t* out;
  float* lse;
  float* part_o;    // rows of head_dim fp32 values, normalised per share; the order of the rows: part_row()
  float* part_lse;  // one fp32 value per row, log2 domain; -inf: no key seen; NaN where the row's sum is NaN
  uint32_t* status;
  int64_t q_batch_stride, q_head_stride;
  int64_t o_batch_stride, o_head_stride;
  int heads_q, heads_kv, group, chunks, len_k, head_dim, rows;  // rows: query heads per unit, min(group, 16)
  int units, tiles_per_unit, grid;
  int num_splits, tiles_per_split;  // num_splits > 0: the caller fixed the shares, CTA = (unit, split)
  float scale_log2;
  int f16;
};

// Tiles [first, last) of the list (tile = unit * tiles_per_unit + tile in unit) that CTA `i` works on.
__host__ __device__ __forceinline__ void cta_share(const DecodeParams& p, int i, int64_t& first, int64_t& last) {
  if (p.num_splits > 0) {
    const int u = i / p.num_splits, sp = i - u * p.num_splits;
    const int lo = sp * p.tiles_per_split, hi = lo + p.tiles_per_split;
    first = static_cast<int64_t>(u) * p.tiles_per_unit + (lo < p.tiles_per_unit ? lo : p.tiles_per_unit);
    last = static_cast<int64_t>(u) * p.tiles_per_unit + (hi < p.tiles_per_unit ? hi : p.tiles_per_unit);
  } else {
    const int64_t total = static_cast<int64_t>(p.units) * p.tiles_per_unit;
    first = i * total / p.grid;
    last = (i + 1) * total / p.grid;
  }
}

// The CTA whose share holds `tile` (equal shares only).
__device__ __forceinline__ int cta_of(const DecodeParams& p, int64_t tile) {
  const int64_t total = static_cast<int64_t>(p.units) * p.tiles_per_unit;
  return static_cast<int>(((tile + 1) * p.grid - 1) / total);
}

// Row of the partial results for one query head: with fixed splits [batch * heads_q][splits]; with equal shares two slots of
// `rows` heads per CTA, slot 0 for the unit its share begins in and slot 1 for the unit it ends in (`r`: head in the unit).
__device__ __forceinline__ int64_t part_row(const DecodeParams& p, int cta, int slot, int head_row, int r) {
  if (p.num_splits > 0) return static_cast<int64_t>(head_row) * p.num_splits + cta % p.num_splits;
  return (2 * static_cast<int64_t>(cta) + slot) * p.rows + r;
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

template <bool kF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                          uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (kF16)
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Same MMA when only fragment rows 0-7 carry query heads: rows 8-15 of A are zero, so their
// accumulators are constants and need no live registers.
template <bool kF16>
__device__ __forceinline__ void mma_16816_lo(float& c0, float& c1, uint32_t a0, uint32_t a2,
                                             uint32_t b0, uint32_t b1) {
  float d2, d3;
  if constexpr (kF16)
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %5}, "
        "{%7, %8}, {%0, %1, %9, %9};"
        : "+f"(c0), "+f"(c1), "=f"(d2), "=f"(d3)
        : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %5}, "
        "{%7, %8}, {%0, %1, %9, %9};"
        : "+f"(c0), "+f"(c1), "=f"(d2), "=f"(d3)
        : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}

template <bool kHi, bool kF16>
__device__ __forceinline__ void mma_rows(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kHi) mma_16816<kF16>(c, a[0], a[1], a[2], a[3], b0, b1);
  else mma_16816_lo<kF16>(c[0], c[1], a[0], a[2], b0, b1);
}

__device__ __forceinline__ float quad_max(float x) {
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
  return x;
}

__device__ __forceinline__ float quad_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x;
}

// Stages of each warp's ring: what lets two CTAs share an SM's 228 KB.
template <bool kHi, int kD>
__host__ __device__ constexpr int decode_stages() { return (kHi ? 2 : 3) * (128 / kD); }
template <int kD>
__host__ __device__ constexpr uint32_t decode_stage_bytes() { return 2u * (kD / 64) * kBoxBytes; }
// per merging warp: accumulators in fragment order [value][lane], then row maxima and sums
template <bool kHi, int kD>
__host__ __device__ constexpr int decode_merge_floats() { return ((kHi ? 4 : 2) * (kD / 8) + (kHi ? 4 : 2)) * 32; }
template <bool kHi, int kD>
__host__ __device__ constexpr uint32_t decode_smem_bytes() {
  return 1024 + kDecWarps * decode_stages<kHi, kD>() * decode_stage_bytes<kD>() +
         (kDecWarps - 1) * decode_merge_floats<kHi, kD>() * 4 + kDecWarps * decode_stages<kHi, kD>() * 8 + 16;
}

// kHi: a unit has more than 8 query heads, so fragment rows 8-15 are in use too.
template <bool kHi, int kD, bool kF16, bool kCluster>
__global__ void __launch_bounds__(kDecThreads, kCtasPerSm)
decode_splitkv_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const DecodeParams p) {
  constexpr int kKSteps = kD / 16;   // MMAs over head_dim for Q K^T
  constexpr int kNBlocks = kD / 8;   // 8-column output blocks of P V
  constexpr int kBoxes = kD / 64;    // 64-column boxes per operand and stage
  constexpr int kSt = decode_stages<kHi, kD>();
  constexpr uint32_t kStageBytes = decode_stage_bytes<kD>();
  constexpr int kMergeFloats = decode_merge_floats<kHi, kD>();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  float* merge = reinterpret_cast<float*>(smem_raw + (base - raw_addr) + kDecWarps * kSt * kStageBytes);
  // kCluster: this CTA's part, [16 heads][kD] and their log2 sums, in the ring, which is idle by then
  float* cl_o = reinterpret_cast<float*>(smem_raw + (base - raw_addr));
  float* cl_lse = cl_o + 16 * kD;
  static_assert(16 * (kD + 1) * 4 <= kDecWarps * kSt * kStageBytes, "a part does not fit the ring");
  const uint32_t bars = smem_u32(merge + (kDecWarps - 1) * kMergeFloats);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(merge + (kDecWarps - 1) * kMergeFloats + kDecWarps * kSt * 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2;  // fragment row (query head within the unit) / key within a block of 8
  const int t = lane & 3;
  const uint32_t ring = base + warp * (kSt * kStageBytes);
  const uint32_t bar = bars + warp * (kSt * 8);

  // the merge kernel behind this one may be launched as soon as every CTA is running (it waits for this grid's results)
  if (threadIdx.x == 0) launch_dependents();

  int64_t first, last;
  cta_share(p, blockIdx.x, first, last);
  const int n_tiles = static_cast<int>(last - first);
  const int unit0 = static_cast<int>(first / p.tiles_per_unit);
  const int tile0 = static_cast<int>(first - static_cast<int64_t>(unit0) * p.tiles_per_unit);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kDecWarps * kSt; ++i) mbar_init(bars + 8 * i, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (elect_one()) {
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  wait_for_previous_grid();  // launched under its tail (launch_split)
  __syncthreads();

  // ---- the load side of the warp's ring: its own step, tile and unit, kSt steps ahead of the arithmetic
  int ld_unit = unit0, ld_tile = tile0, ld_step = 0;
  int ld_b, ld_hk;
  auto load_unit = [&]() {
    const int hc = ld_unit / p.chunks;
    ld_b = hc / p.heads_kv;
    ld_hk = hc - ld_b * p.heads_kv;
  };
  load_unit();
  auto issue_load = [&]() {  // called by one lane
    const uint32_t st = ld_step % kSt;
    const uint32_t dst = ring + st * kStageBytes, full = bar + 8 * st;
    const int row = ld_tile * kTileKeys + warp * kKeysPerStep;
    mbar_arrive_expect_tx(full, kStageBytes);
#pragma unroll
    for (int c = 0; c < kBoxes; ++c) tma_load_4d(dst + c * kBoxBytes, &tm_k, full, c * 64, row, ld_hk, ld_b);
#pragma unroll
    for (int c = 0; c < kBoxes; ++c) tma_load_4d(dst + (kBoxes + c) * kBoxBytes, &tm_v, full, c * 64, row, ld_hk, ld_b);
  };
  auto next_load = [&]() {
    ++ld_step;
    if (++ld_tile == p.tiles_per_unit) {
      ld_tile = 0;
      ++ld_unit;
      load_unit();
    }
  };
  for (int i = 0; i < kSt && i < n_tiles; ++i) {
    if (elect_one()) issue_load();
    next_load();
  }

  // ---- Q fragments of a unit
  uint32_t qa[kKSteps][4], qn[kKSteps][4];
  auto load_q = [&](int unit, uint32_t (&dst)[kKSteps][4]) {
    const int hc = unit / p.chunks, b = hc / p.heads_kv;
    const int head0 = (hc - b * p.heads_kv) * p.group + (unit - hc * p.chunks) * 16;
    const int nheads = min(16, p.group - (unit - hc * p.chunks) * 16);
    const uint16_t* q0 = p.q + b * p.q_batch_stride + (head0 + g) * p.q_head_stride + 2 * t;
    const uint16_t* q8 = q0 + 8 * p.q_head_stride;
#pragma unroll
    for (int i = 0; i < kKSteps; ++i) {
      dst[i][0] = dst[i][1] = dst[i][2] = dst[i][3] = 0u;
      if (g < nheads) {
        dst[i][0] = *reinterpret_cast<const uint32_t*>(q0 + i * 16);      // row g,   k 2t..2t+1
        dst[i][2] = *reinterpret_cast<const uint32_t*>(q0 + i * 16 + 8);  // row g,   k 2t+8..2t+9
      }
      if (kHi && g + 8 < nheads) {
        dst[i][1] = *reinterpret_cast<const uint32_t*>(q8 + i * 16);
        dst[i][3] = *reinterpret_cast<const uint32_t*>(q8 + i * 16 + 8);
      }
    }
  };
  if (n_tiles > 0) load_q(unit0, qn);

  const float c = p.scale_log2;
  // ldmatrix row addresses inside a box: this lane's row of each of the four 8x8 matrices
  const int mrow = lane & 7, mat = lane >> 3;
  bool ok = true;
  int step = 0;
  for (int unit = unit0, tile = tile0; step < n_tiles; ++unit, tile = 0) {
    const int seg_tiles = min(n_tiles - step, p.tiles_per_unit - tile);
    const bool whole = seg_tiles == p.tiles_per_unit && p.num_splits <= 1;
#pragma unroll
    for (int i = 0; i < kKSteps; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) qa[i][j] = qn[i][j];
    if (step + seg_tiles < n_tiles) load_q(unit + 1, qn);  // in flight under this unit's tiles

    float o[kNBlocks][4];
#pragma unroll
    for (int nb = 0; nb < kNBlocks; ++nb) o[nb][0] = o[nb][1] = o[nb][2] = o[nb][3] = 0.f;
    float m_lo = -INFINITY, m_hi = -INFINITY;  // running max (log2 domain) of rows g and g+8
    float l_lo = 0.f, l_hi = 0.f;              // this thread's share of the running sums

    for (int i = 0; i < seg_tiles; ++i, ++step) {
      const uint32_t st = step % kSt;
      const uint32_t k_smem = ring + st * kStageBytes, v_smem = k_smem + kBoxes * kBoxBytes;
      if (ok) ok = mbar_wait(bar + 8 * st, (step / kSt) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);

      // ---- S = Q K^T for two blocks of 8 keys
      float s[2][4];
#pragma unroll
      for (int blk = 0; blk < 2; ++blk) {
        s[blk][0] = s[blk][1] = s[blk][2] = s[blk][3] = 0.f;
#pragma unroll
        for (int ch = 0; ch < kD / 8; ch += 4) {  // four 16-byte chunks of 8 keys = the B fragments of two K steps
          uint32_t kf[4];
          const int chunk = ch + mat;
          ldmatrix_x4(k_smem + (chunk >> 3) * kBoxBytes + (blk * 8 + mrow) * kBoxRowBytes + (((chunk & 7) ^ mrow) << 4), kf);
          mma_rows<kHi, kF16>(s[blk], qa[ch / 2], kf[0], kf[1]);
          mma_rows<kHi, kF16>(s[blk], qa[ch / 2 + 1], kf[2], kf[3]);
        }
      }

      // ---- mask the tail, online softmax (thread holds keys key0 + blk*8 + 2t + {0,1})
      const int key0 = (tile + i) * kTileKeys + warp * kKeysPerStep;
      if (key0 + kKeysPerStep > p.len_k) {
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          const int kk = key0 + blk * 8 + 2 * t;
          if (kk >= p.len_k) { s[blk][0] = -INFINITY; s[blk][2] = -INFINITY; }
          if (kk + 1 >= p.len_k) { s[blk][1] = -INFINITY; s[blk][3] = -INFINITY; }
        }
      }
      // The exponents are taken against this tile's own maximum and the tile's sums join the running ones with an fp32 factor: the
      // largest of every 16 keys is then a P of exactly 1. Against a running maximum, which a share of hundreds of tiles rarely
      // renews, the 16-bit P of all large weights are rounded: error against 64 bits (bf16, Lk 32768) 2.21e-3 instead of 1.95e-3.
      // The kernel waits for HBM (a fifth of its issue slots are used), so the factors cost no time: B 64 Lk 32768 1218 us both ways.
      const float t_lo = quad_max(fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]))) * c;
      const float t_hi = kHi ? quad_max(fmaxf(fmaxf(s[0][2], s[0][3]), fmaxf(s[1][2], s[1][3]))) * c : -INFINITY;
      const float mn_lo = fmaxf(m_lo, t_lo), mn_hi = fmaxf(m_hi, t_hi);
      // a row without a key so far (maximum -inf) has o = l = 0 and a tile of zeros: any finite factor will do
      const float a_lo = (mn_lo == -INFINITY) ? 1.f : ex2_approx(m_lo - mn_lo), b_lo = (mn_lo == -INFINITY) ? 1.f : ex2_approx(t_lo - mn_lo);
      const float a_hi = (!kHi || mn_hi == -INFINITY) ? 1.f : ex2_approx(m_hi - mn_hi);
      const float b_hi = (!kHi || mn_hi == -INFINITY) ? 1.f : ex2_approx(t_hi - mn_hi);
      m_lo = mn_lo;
      m_hi = mn_hi;
      const float u_lo = (t_lo == -INFINITY) ? 0.f : t_lo, u_hi = (t_hi == -INFINITY) ? 0.f : t_hi;
      float pr[2][4], lt_lo = 0.f, lt_hi = 0.f;
#pragma unroll
      for (int blk = 0; blk < 2; ++blk) {
        pr[blk][0] = ex2_approx(fmaf(s[blk][0], c, -u_lo));
        pr[blk][1] = ex2_approx(fmaf(s[blk][1], c, -u_lo));
        pr[blk][2] = kHi ? ex2_approx(fmaf(s[blk][2], c, -u_hi)) : 0.f;
        pr[blk][3] = kHi ? ex2_approx(fmaf(s[blk][3], c, -u_hi)) : 0.f;
        lt_lo += pr[blk][0] + pr[blk][1];
        lt_hi += pr[blk][2] + pr[blk][3];
      }
      l_lo = fmaf(lt_lo, b_lo, l_lo * a_lo);
      l_hi = fmaf(lt_hi, b_hi, l_hi * a_hi);
      uint32_t pa[4];
      pa[0] = pack_16x2<kF16>(pr[0][0], pr[0][1]);  // row g,   keys 2t, 2t+1
      pa[1] = pack_16x2<kF16>(pr[0][2], pr[0][3]);  // row g+8
      pa[2] = pack_16x2<kF16>(pr[1][0], pr[1][1]);  // row g,   keys 8+2t, 9+2t
      pa[3] = pack_16x2<kF16>(pr[1][2], pr[1][3]);  // row g+8

      // ---- O += P V: matrices (keys 0-7, chunk), (keys 8-15, chunk), the same for the next chunk
#pragma unroll
      for (int ch = 0; ch < kD / 8; ch += 2) {
        uint32_t vf[4];
        const int chunk = ch + (mat >> 1);
        ldmatrix_x4_trans(v_smem + (chunk >> 3) * kBoxBytes + ((mat & 1) * 8 + mrow) * kBoxRowBytes + (((chunk & 7) ^ mrow) << 4), vf);
        float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        mma_rows<kHi, kF16>(d[0], pa, vf[0], vf[1]);
        mma_rows<kHi, kF16>(d[1], pa, vf[2], vf[3]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          o[ch + e][0] = fmaf(d[e][0], b_lo, o[ch + e][0] * a_lo);
          o[ch + e][1] = fmaf(d[e][1], b_lo, o[ch + e][1] * a_lo);
          if (kHi) {
            o[ch + e][2] = fmaf(d[e][2], b_hi, o[ch + e][2] * a_hi);
            o[ch + e][3] = fmaf(d[e][3], b_hi, o[ch + e][3] * a_hi);
          }
        }
      }
      // the stage has been read by every lane: refill it
      __syncwarp();
      if (ld_step < n_tiles) {
        if (ok && elect_one()) issue_load();
        next_load();
      }
    }

    // ---- merge the four warps: 1-3 hand their state over in fragment order, warp 0 folds it into its own
    l_lo = quad_sum(l_lo);
    l_hi = quad_sum(l_hi);
    __syncthreads();  // warp 0 has read what the previous unit left here
    if (warp > 0) {
      float* dst = merge + (warp - 1) * kMergeFloats + lane;
#pragma unroll
      for (int nb = 0; nb < kNBlocks; ++nb) {
#pragma unroll
        for (int e = 0; e < (kHi ? 4 : 2); ++e) dst[(nb * (kHi ? 4 : 2) + e) * 32] = o[nb][e];
      }
      dst += kNBlocks * (kHi ? 4 : 2) * 32;
      dst[0] = m_lo;
      dst[32] = l_lo;
      if (kHi) {
        dst[64] = m_hi;
        dst[96] = l_hi;
      }
    }
    __syncthreads();
    if (warp == 0) {
      constexpr int kTail = kNBlocks * (kHi ? 4 : 2) * 32;
      float mm_lo = m_lo, mm_hi = m_hi;
#pragma unroll
      for (int w = 0; w < kDecWarps - 1; ++w) {
        mm_lo = fmaxf(mm_lo, merge[w * kMergeFloats + kTail + lane]);
        if (kHi) mm_hi = fmaxf(mm_hi, merge[w * kMergeFloats + kTail + 64 + lane]);
      }
      auto weight = [](float m, float mm) { return (m == -INFINITY) ? 0.f : ex2_approx(m - mm); };
      float f_lo = weight(m_lo, mm_lo), f_hi = kHi ? weight(m_hi, mm_hi) : 0.f;
      l_lo *= f_lo;
      l_hi *= f_hi;
#pragma unroll
      for (int nb = 0; nb < kNBlocks; ++nb) {
        o[nb][0] *= f_lo;
        o[nb][1] *= f_lo;
        o[nb][2] *= f_hi;
        o[nb][3] *= f_hi;
      }
#pragma unroll
      for (int w = 0; w < kDecWarps - 1; ++w) {
        const float* src = merge + w * kMergeFloats + lane;
        f_lo = weight(src[kTail], mm_lo);
        l_lo += src[kTail + 32] * f_lo;
        if (kHi) {
          f_hi = weight(src[kTail + 64], mm_hi);
          l_hi += src[kTail + 96] * f_hi;
        }
#pragma unroll
        for (int nb = 0; nb < kNBlocks; ++nb) {
#pragma unroll
          for (int e = 0; e < (kHi ? 4 : 2); ++e) o[nb][e] += src[(nb * (kHi ? 4 : 2) + e) * 32] * (e < 2 ? f_lo : f_hi);
        }
      }
      const int hc = unit / p.chunks, b = hc / p.heads_kv;
      const int head0 = (hc - b * p.heads_kv) * p.group + (unit - hc * p.chunks) * 16;
      const int nheads = min(16, p.group - (unit - hc * p.chunks) * 16);
#pragma unroll
      for (int hi = 0; hi < (kHi ? 2 : 1); ++hi) {
        const int r = g + 8 * hi;
        if (r >= nheads) continue;
        const float l = hi ? l_hi : l_lo, mm = hi ? mm_hi : mm_lo;
        const float inv = (l > 0.f) ? 1.f / l : 0.f;
        const float lse2 = (l == 0.f) ? -INFINITY : mm + log2f(l);  // a NaN sum stays visible to the merge
        if constexpr (kCluster) {
          float* dst = cl_o + r * kD + 2 * t;
#pragma unroll
          for (int nb = 0; nb < kNBlocks; ++nb)
            *reinterpret_cast<float2*>(dst + nb * 8) = make_float2(o[nb][2 * hi] * inv, o[nb][2 * hi + 1] * inv);
          if (t == 0) cl_lse[r] = lse2;
        } else if (whole) {
          uint16_t* dst = p.out + b * p.o_batch_stride + (head0 + r) * p.o_head_stride + 2 * t;
#pragma unroll
          for (int nb = 0; nb < kNBlocks; ++nb)
            *reinterpret_cast<uint32_t*>(dst + nb * 8) = pack_16x2<kF16>(o[nb][2 * hi] * inv, o[nb][2 * hi + 1] * inv);
          if (t == 0) p.lse[static_cast<int64_t>(b) * p.heads_q + head0 + r] = (l > 0.f) ? lse2 * 0.6931471805599453f : INFINITY;
        } else {
          const int64_t row = part_row(p, blockIdx.x, unit == unit0 ? 0 : 1, b * p.heads_q + head0 + r, r);
          float* dst = p.part_o + row * kD + 2 * t;
#pragma unroll
          for (int nb = 0; nb < kNBlocks; ++nb)
            *reinterpret_cast<float2*>(dst + nb * 8) = make_float2(o[nb][2 * hi] * inv, o[nb][2 * hi + 1] * inv);
          if (t == 0) p.part_lse[row] = lse2;
        }
      }
    }
  }
  if constexpr (kCluster) {
    // ---- merge over the cluster: every CTA takes a share of the columns of all parts, out of the others' shared memory
    const int size = p.num_splits, rank = static_cast<int>(blockIdx.x) % size;
    if (n_tiles == 0 && threadIdx.x < 16) cl_lse[threadIdx.x] = -INFINITY;
    cluster_sync();
    const int u = blockIdx.x / size, hc = u / p.chunks, b = hc / p.heads_kv;
    const int head0 = (hc - b * p.heads_kv) * p.group + (u - hc * p.chunks) * 16;
    const int nheads = min(16, p.group - (u - hc * p.chunks) * 16);
    const int pairs = kD / 2 / size;  // column pairs of this CTA
    for (int e = threadIdx.x; e < nheads * pairs; e += kDecThreads) {
      const int r = e / pairs, col = 2 * (rank * pairs + e - r * pairs);
      const uint32_t o_addr = smem_u32(cl_o + r * kD + col), lse_addr = smem_u32(cl_lse + r);
      float ls[kMaxCluster];
      float2 x[kMaxCluster];
#pragma unroll
      for (int j = 0; j < kMaxCluster; ++j) {
        ls[j] = -INFINITY;
        x[j] = make_float2(0.f, 0.f);
        if (j < size) {
          ls[j] = cluster_ld_f32(lse_addr, j);
          if (ls[j] != -INFINITY) x[j] = cluster_ld_f32x2(o_addr, j);  // an empty part has written no row; a NaN part is not one
        }
      }
      float m = ls[0];
#pragma unroll
      for (int j = 1; j < kMaxCluster; ++j) m = fmaxf(m, ls[j]);
      float l = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll
      for (int j = 0; j < kMaxCluster; ++j) {
        const float w = (ls[j] == -INFINITY) ? 0.f : exp2f(ls[j] - m);
        l += w;
        v0 += w * x[j].x;
        v1 += w * x[j].y;
      }
      const float inv = (l > 0.f) ? 1.f / l : 0.f;
      *reinterpret_cast<uint32_t*>(p.out + b * p.o_batch_stride + (head0 + r) * p.o_head_stride + col) = pack_16x2<kF16>(v0 * inv, v1 * inv);
      if (col == 0) p.lse[static_cast<int64_t>(b) * p.heads_q + head0 + r] = (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : INFINITY;
    }
    cluster_sync();  // the others have read this CTA's part
  }
  // a fixed split without keys (more splits than tiles): its merge partner finds an empty part
  if (!kCluster && n_tiles == 0 && p.num_splits > 1) {
    const int u = blockIdx.x / p.num_splits, hc = u / p.chunks, b = hc / p.heads_kv;
    const int chunk = u - hc * p.chunks;
    if (static_cast<int>(threadIdx.x) < min(16, p.group - chunk * 16))
      p.part_lse[part_row(p, blockIdx.x, 0, b * p.heads_q + (hc - b * p.heads_kv) * p.group + chunk * 16 + threadIdx.x, 0)] = -INFINITY;
  }
  if (lane == 0) drain_after_abort(abort_flag);
  if (threadIdx.x == 0 && *abort_flag != 0) atomicExch(p.status, static_cast<uint32_t>(SDPA_B200_DEVICE_TIMEOUT));
}

// Merges the parts of the units that several CTAs worked on: one CTA of four warps per (batch, query head), each warp a
// quarter of the parts, lanes over head_dim.
template <int kD>
__global__ void __launch_bounds__(128) decode_combine_kernel(const DecodeParams p) {
  __shared__ float sm_o[3][kD], sm_m[4], sm_l[4];
  if (threadIdx.x == 0) launch_dependents();
  const int row = blockIdx.x;  // batch * heads_q + query head
  const int b = row / p.heads_q, hq = row - b * p.heads_q;
  const int hk = hq / p.group, in_group = hq - hk * p.group;
  const int unit = (b * p.heads_kv + hk) * p.chunks + in_group / 16, r = in_group % 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int c0, c1;  // CTAs [c0, c1] hold the unit's tiles
  const int64_t u0 = static_cast<int64_t>(unit) * p.tiles_per_unit;
  if (p.num_splits > 0) {
    c0 = unit * p.num_splits;
    c1 = c0 + p.num_splits - 1;
  } else {
    c0 = cta_of(p, u0);
    c1 = cta_of(p, u0 + p.tiles_per_unit - 1);
  }
  wait_for_previous_grid();  // the parts are written
  if (c0 == c1) return;  // one CTA had all of it and wrote the result itself
  const int64_t total = static_cast<int64_t>(p.units) * p.tiles_per_unit;
  // the unit's part of CTA c is its slot 0 unless c began in an earlier unit (only c0 can have)
  const int first_slot = (p.num_splits == 0 && c0 * total / p.grid < u0) ? 1 : 0;

  float m = -INFINITY, l = 0.f;
  constexpr int kPer = kD / 32;  // floats per lane
  float acc[kPer];
#pragma unroll
  for (int e = 0; e < kPer; ++e) acc[e] = 0.f;
  for (int c = c0 + warp * 4; c <= c1; c += 16) {
    float ls[4], x[4][kPer];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool have = c + j <= c1;
      const int cj = have ? c + j : c;
      const int64_t pr = part_row(p, cj, cj == c0 ? first_slot : 0, row, r);
      ls[j] = have ? p.part_lse[pr] : -INFINITY;
#pragma unroll
      for (int e = 0; e < kPer; ++e) x[j][e] = (ls[j] == -INFINITY) ? 0.f : p.part_o[pr * kD + e * 32 + lane];
    }
    // empty parts are left out by their own weight: a NaN part is not one, and fmaxf does not return it
    if (ls[0] == -INFINITY && ls[1] == -INFINITY && ls[2] == -INFINITY && ls[3] == -INFINITY) continue;
    const float mn = fmaxf(fmaxf(fmaxf(ls[0], ls[1]), fmaxf(ls[2], ls[3])), m);
    const float a = (m == -INFINITY) ? 1.f : exp2f(m - mn);  // nothing summed yet, or NaN
    l *= a;
#pragma unroll
    for (int e = 0; e < kPer; ++e) acc[e] *= a;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float w = (ls[j] == -INFINITY) ? 0.f : exp2f(ls[j] - mn);
      l += w;
#pragma unroll
      for (int e = 0; e < kPer; ++e) acc[e] += w * x[j][e];
    }
    m = mn;
  }
  if (lane == 0) {
    sm_m[warp] = m;
    sm_l[warp] = l;
  }
  if (warp > 0) {
#pragma unroll
    for (int e = 0; e < kPer; ++e) sm_o[warp - 1][e * 32 + lane] = acc[e];
  }
  __syncthreads();
  if (warp != 0) return;
  const float mm = fmaxf(fmaxf(sm_m[0], sm_m[1]), fmaxf(sm_m[2], sm_m[3]));
  float sum = 0.f, f[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    f[w] = (sm_m[w] == -INFINITY) ? 0.f : exp2f(sm_m[w] - mm);
    sum += sm_l[w] * f[w];  // 0 * NaN is NaN: a quarter of NaN parts only counts as well
  }
  const float inv = (sum > 0.f) ? 1.f / sum : 0.f;
  uint16_t* dst = p.out + b * p.o_batch_stride + hq * p.o_head_stride;
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    float v = acc[e] * f[0];
#pragma unroll
    for (int w = 1; w < 4; ++w) v += sm_o[w - 1][e * 32 + lane] * f[w];
    dst[e * 32 + lane] = p.f16 ? to_16<true>(v * inv) : to_16<false>(v * inv);
  }
  if (lane == 0) p.lse[row] = (sum > 0.f) ? (mm + log2f(sum)) * 0.6931471805599453f : INFINITY;
}

// How the keys are shared out: by the caller's num_splits, or in equal shares over one wave of CTAs.
void plan_decode(const sdpa_b200_params& p, int sms, DecodeParams& d) {
  d.group = p.heads_q / p.heads_kv;
  d.chunks = (d.group + 15) / 16;
  d.rows = d.group < 16 ? d.group : 16;
  d.units = p.batch * p.heads_kv * d.chunks;
  d.tiles_per_unit = (p.max_seqlen_k + kTileKeys - 1) / kTileKeys;
  d.num_splits = 0;
  d.tiles_per_split = 0;
  if (p.num_splits > 0) {
    d.num_splits = p.num_splits > kMaxSplits ? kMaxSplits : p.num_splits;
    d.tiles_per_split = (d.tiles_per_unit + d.num_splits - 1) / d.num_splits;
    d.grid = d.units * d.num_splits;
  } else {
    const int64_t total = static_cast<int64_t>(d.units) * d.tiles_per_unit;
    const int64_t wave = static_cast<int64_t>(kCtasPerSm) * sms;
    d.grid = static_cast<int>(total < wave ? total : wave);
  }
}

// CTAs per unit of a launch that needs no merge kernel: 1 (units stay whole), or a cluster of 2 to 8 that merges in shared memory; 0: equal shares
// over one wave and the merge kernel, whose second launch costs about 3 us. Figures in us, calls back to back, H32/8 D128 unless said, equal
// shares | so:
//  * One wave of clusters, where its longest share is not much longer than an equal one: B1 Lk 1000 8.8 | 6.6, Lk 2000 8.7 | 7.9 (but Lk 4000 8.8 |
//    10.1), B8 Lk 1000 10.2 | 8.8, Lk 4096 27.3 | 26.0, B16 Lk 1000 12.5 | 11.0. Clusters of 8 find room for 256 CTAs at once, not for 296: B3
//    H12/12 Lk 4000 in 288 CTAs 13.1 | 20.4; so for fours too, which come after them.
//  * One nearly full wave of whole units, up to where a second wave of clusters has long enough shares: B32 Lk 500 12.5 | 9.1, B30 Lk 300 D64 9.0 | 6.3, B34 Lk 900
//    26.4 | 23.1, B30 Lk 3900 80.1 | 78.5 (192 units, B24 Lk 3000 51.8 | 52.4).
//  * Several waves whose last one has at least 160 of 296 CTAs. The hardware deals them out, where the slowest SM ends an equal share: B64 Lk 32768
//    1249 | 1164, Lk 1500 66.6 | 59.7, Lk 300 16.1 | 13.2 (last wave nearly empty: B30 H12/12 Lk 2000 60.9 | 63.7, B44 Lk 300 11.8 | 12.3; many waves of a
//    few tiles: B64 H32/32 Lk 64 19.0 | 22.6).
//  * The same in clusters of two or four. A wave of clusters costs 3 to 4 us, so those take long shares only: B32 Lk 16384 in twos 316 | 300, B57 H16/4 Lk
//    9000 162 | 152, B16 Lk 16384 in fours 316 | 310, B30 H16/4 Lk 18000 170 | 160, D64 91.0 | 86.5 (B16 Lk 1000 in fours 12.5 | 16.6; with 104 CTAs in the last wave, B25
//    H16/4 Lk 8300 D64 39.6 | 44.6, with 80, B42 61.9 | 67.1; in shares of half the bytes, B18 H12/12
//    Lk 9684 D64 89.7 | 94.3). Not in eights, which find room for 256 CTAs: two full waves of those, B8 Lk 20000 D64 57.2 | 60.0, 2.25 of them, B9 Lk 17000 57 | 65.
int cluster_size(const DecodeParams& d) {
  constexpr int kWave = kCtasPerSm * 148;
  const int64_t units = d.units;
  const int tiles = d.tiles_per_unit;
  for (int size = kMaxCluster; size > 1; size /= 2) {
    if (size > tiles || units * size > (size > 2 ? 256 : kWave)) continue;
    if ((tiles + size - 1) / size - static_cast<double>(units) * tiles / kWave <= 3.5) return size;
    break;
  }
  if (units <= kWave && units >= kWave * 4 / 5 && tiles < 63) return 1;
  for (int size = 1; size <= 4; size *= 2) {
    const int64_t ctas = units * size, last = ctas % kWave;
    const int least = size == 4 && d.head_dim == 64 ? 64 : 32;  // tiles of a cluster's share
    if (ctas >= kWave && (last == 0 || last >= 160) && (size == 1 ? tiles > ctas / kWave : (tiles + size - 1) / size >= least)) return size;
  }
  return 0;
}

// Rows of partial results the workspace must hold (0: every unit stays whole).
size_t partial_rows(const sdpa_b200_params& p, const DecodeParams& d) {
  if (d.num_splits == 1) return 0;
  if (d.num_splits > 1) return static_cast<size_t>(p.batch) * p.heads_q * d.num_splits;
  return static_cast<size_t>(d.grid) * 2 * d.rows;
}

constexpr int kPlanSms = 160;  // workspace sizes do not ask the device: an upper bound of its SMs (148)

}  // namespace

size_t decode_workspace_bytes(const sdpa_b200_params& p) {
  DecodeParams d;
  plan_decode(p, kPlanSms, d);
  const size_t rows = partial_rows(p, d);
  return rows == 0 ? 0 : rows * sizeof(float) * (p.head_dim + 1) + 256;
}

namespace {

template <bool kHi, int kD, bool kF16, bool kCluster = false>
cudaError_t launch_split(const CUtensorMap& tm_k, const CUtensorMap& tm_v, const DecodeParams& d, bool overlap, cudaStream_t stream) {
  constexpr uint32_t kSmem = decode_smem_bytes<kHi, kD>();
  auto kernel = decode_splitkv_kernel<kHi, kD, kF16, kCluster>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (err != cudaSuccess) return err;
  return launch_behind(kernel, dim3(d.grid), kDecThreads, kSmem, stream, overlap, kCluster ? d.num_splits : 1, tm_k, tm_v, d);
}

template <int kD>
cudaError_t launch_combine(const DecodeParams& d, int rows, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows);
  cfg.blockDim = dim3(128);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, decode_combine_kernel<kD>, d);
}

// The split kernel and, where units are shared between CTAs, the merge kernel. Partial results go to `scratch`
// (partial_rows() rows of head_dim + 1 floats).
int launch_decode(const sdpa_b200_params& p, DecodeParams& d, float* scratch, uint32_t* status, const char* who, cudaStream_t stream) {
  const bool f16 = p.dtype == SDPA_B200_F16;
  const size_t rows = partial_rows(p, d);
  d.q = static_cast<const uint16_t*>(p.q);
  d.out = static_cast<uint16_t*>(p.out);
  d.lse = p.lse;
  d.part_o = scratch;
  d.part_lse = scratch + rows * p.head_dim;
  d.status = status;
  d.q_batch_stride = p.q_batch_stride;
  d.q_head_stride = p.q_head_stride;
  d.o_batch_stride = p.o_batch_stride;
  d.o_head_stride = p.o_head_stride;
  d.heads_q = p.heads_q;
  d.heads_kv = p.heads_kv;
  d.len_k = p.max_seqlen_k;
  d.head_dim = p.head_dim;
  d.scale_log2 = p.softmax_scale * 1.4426950408889634f;
  d.f16 = f16;
  CUtensorMap tm_k, tm_v;
  // the stride of a single head means nothing and may be any number, but the tensor map wants a legal one
  const bool one_head = p.heads_kv == 1;
  int st = make_tensor_map_16(f16, &tm_k, p.k, p.head_dim, p.max_seqlen_k, p.heads_kv, p.batch, p.k_row_stride,
                              one_head ? p.k_row_stride : p.k_head_stride, p.k_batch_stride, kKeysPerStep);
  if (st != SDPA_B200_OK) return st;
  st = make_tensor_map_16(f16, &tm_v, p.v, p.head_dim, p.max_seqlen_k, p.heads_kv, p.batch, p.v_row_stride,
                          one_head ? p.v_row_stride : p.v_head_stride, p.v_batch_stride, kKeysPerStep);
  if (st != SDPA_B200_OK) return st;
  const int cluster = p.num_splits > 0 ? 0 : cluster_size(d);
  if (cluster > 0) {
    d.num_splits = cluster;
    d.tiles_per_split = (d.tiles_per_unit + cluster - 1) / cluster;
    d.grid = d.units * cluster;
  }
  const bool hi = d.rows > 8;
  // under the tail of whatever is in front, unless that is the launch that clears the status word (calls back to back: B64 H32/8 Lk 84 D64
  // 12.3 us -> 9.7, B8 Lk 4096 D128 29.7 -> 27.4, B1 Lk 1000 9.0 -> 8.6)
  // But not a fixed split into long shares with CTAs for more than a quarter of the SMs (half of them, where the merge kernel stands between two such grids) and fewer than
  // fill them twice: those that start early find part of the SMs taken, share others in pairs and stream at half the rate to the end (calls back to back, early | plain start:
  // H16/16, Lk 5857, one split, D64 B4 43.4 | 37.4, B9 44.9 | 40.1, B12 51.9 | 49.3, D128 B6 58.3 | 52.2, B5 H8/8 Lk 9000 D64, 40 CTAs, 62.8 | 55.3, three splits, B2 18.8 | 18.5; but one
  // split, 32 CTAs, B2 H16/16 Lk 3000 D64 19.4 | 20.8, three, 48 CTAs, B1 Lk 9000 D64 22.2 | 24.6, four, 23 tiles, B2 Lk 5857 15.4 | 16.4).
  const bool pairs_up = p.num_splits > 0 && d.tiles_per_split >= 28 && d.grid > (p.num_splits > 1 ? 74 : 37) && d.grid < kCtasPerSm * 148;
  const bool overlap = p.device_status != nullptr && !pairs_up;
  cudaError_t err;
  auto launch = [&](auto hi_tag, auto dim_tag, auto f16_tag) {
    constexpr bool kHi = decltype(hi_tag)::value, kF16 = decltype(f16_tag)::value;
    constexpr int kD = decltype(dim_tag)::value;
    return cluster > 1 ? launch_split<kHi, kD, kF16, true>(tm_k, tm_v, d, overlap, stream) : launch_split<kHi, kD, kF16, false>(tm_k, tm_v, d, overlap, stream);
  };
  auto launch_type = [&](auto hi_tag, auto dim_tag) {
    return f16 ? launch(hi_tag, dim_tag, std::true_type{}) : launch(hi_tag, dim_tag, std::false_type{});
  };
  using Dim64 = std::integral_constant<int, 64>;
  using Dim128 = std::integral_constant<int, 128>;
  if (p.head_dim == 64)
    err = hi ? launch_type(std::true_type{}, Dim64{}) : launch_type(std::false_type{}, Dim64{});
  else
    err = hi ? launch_type(std::true_type{}, Dim128{}) : launch_type(std::false_type{}, Dim128{});
  if (err != cudaSuccess) {
    set_error("%s: launch failed: %s", who, cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  // no merge when the shares' borders coincide with the units'
  const bool shared = cluster > 0 ? false : d.num_splits > 0 ? d.num_splits > 1 : (d.tiles_per_unit > 1 && d.units % d.grid != 0);
  if (shared) {
    const int out_rows = p.batch * p.heads_q;
    err = p.head_dim == 64 ? launch_combine<64>(d, out_rows, stream) : launch_combine<128>(d, out_rows, stream);
    if (err != cudaSuccess) {
      set_error("%s merge: launch failed: %s", who, cudaGetErrorString(err));
      return SDPA_B200_LAUNCH_FAILED;
    }
    count_launch();
  }
  return SDPA_B200_OK;
}

}  // namespace

// What the streaming kernels cannot do; shared by every entry point that launches them.
int check_decode_request(const sdpa_b200_params& p) {
  if (p.cu_seqlens_q != nullptr || p.cu_seqlens_k != nullptr) {
    set_error("the decode kernel takes dense tensors only");
    return SDPA_B200_UNSUPPORTED;
  }
  if (p.max_seqlen_q != 1) {
    set_error("decode kernel needs seqlen_q == 1 (got %d)", p.max_seqlen_q);
    return SDPA_B200_UNSUPPORTED;
  }
  if (p.head_dim != 64 && p.head_dim != 128) {
    set_error("the decode kernel is built for head_dim 64 and 128 only (got %d)", p.head_dim);
    return SDPA_B200_UNSUPPORTED;
  }
  if (p.dropout_p != 0.f || p.keep_rows != nullptr || p.keep_cols != nullptr) {
    set_error("the decode kernel has no dropout");
    return SDPA_B200_UNSUPPORTED;
  }
  if (p.bias != nullptr) {
    set_error("the decode kernel takes no additive bias");
    return SDPA_B200_UNSUPPORTED;
  }
  return SDPA_B200_OK;
}

int launch_fwd_decode(const sdpa_b200_params& p, void* workspace, size_t workspace_bytes,
                      cudaStream_t stream) {
  int st = check_decode_request(p);
  if (st != SDPA_B200_OK) return st;
  const size_t need = decode_workspace_bytes(p);
  if (workspace_bytes < kWorkspaceHeaderBytes + need) {
    set_error("decode workspace too small: %zu < %zu", workspace_bytes, kWorkspaceHeaderBytes + need);
    return SDPA_B200_INVALID_ARG;
  }
  const int sms = sm_count();
  if (sms <= 0 || sms > kPlanSms) {
    set_error("decode: cannot use a device with %d SMs", sms);
    return SDPA_B200_NO_DEVICE;
  }
  DecodeParams d;
  plan_decode(p, sms, d);
  float* scratch = reinterpret_cast<float*>(static_cast<char*>(workspace) + kWorkspaceHeaderBytes);
  uint32_t* status = p.device_status != nullptr ? p.device_status : static_cast<uint32_t*>(workspace);
  return launch_decode(p, d, scratch, status, "decode", stream);
}

}  // namespace sdpa_b200

// ---------------------------------------------------------------------------------------
// Decode without any caller- or library-allocated scratch memory.
//
// Some callers may not allocate device memory at the point where they need attention: code
// running inside a memory-pool callback or an allocator hook, a serving loop whose memory plan
// was frozen at start-up, or a process that has handed the whole device to another allocator.
// For them the split-KV partials live in a fixed array that is part of this library's image;
// every GPU that loads the library carries those SDPA_B200_STATIC_SCRATCH_BYTES until exit.
//
// The array name below is only a host-side handle: in host code it is not a device address and
// must never be handed to a kernel. The real address is asked from the runtime with
// cudaGetSymbolAddress, once per device, with that device current, on the first call made on
// that device (so make that first call outside any stream capture). Nothing is allocated or
// freed here, and no library routine that allocates is called.
//
// All calls on a device share the one array and it keeps whatever the previous call left in
// it. That is harmless for this kernel pair - every (row, split) slot the merge kernel reads is
// written by the split kernel of the same call first, so nothing has to start at zero - but two
// calls whose kernels overlap on the GPU (different streams, no ordering) race on it.
// ---------------------------------------------------------------------------------------
namespace sdpa_b200 {
namespace {

constexpr size_t kStaticHeaderBytes = 256;  // in front of the partials: takes a time-out when the caller gives no status word
static __device__ __align__(256) unsigned char g_decode_static_scratch[SDPA_B200_STATIC_SCRATCH_BYTES + kStaticHeaderBytes];

constexpr int kMaxDevices = 64;
void* g_static_scratch_ptr[kMaxDevices] = {};
std::mutex g_static_scratch_mutex;

// Device address of the static array on the current device (looked up once per device).
int static_scratch_address(void** out) {
  int dev = -1;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    (void)cudaGetLastError();
    set_error("decode_static: cannot identify the current device");
    return SDPA_B200_NO_DEVICE;
  }
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  if (g_static_scratch_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    err = cudaGetSymbolAddress(&ptr, g_decode_static_scratch);
    if (err != cudaSuccess || ptr == nullptr) {
      (void)cudaGetLastError();
      set_error("decode_static: cudaGetSymbolAddress failed on device %d: %s", dev, cudaGetErrorString(err));
      return SDPA_B200_LAUNCH_FAILED;
    }
    g_static_scratch_ptr[dev] = ptr;
  }
  *out = g_static_scratch_ptr[dev];
  return SDPA_B200_OK;
}

}  // namespace
}  // namespace sdpa_b200

extern "C" SDPA_B200_API int sdpa_b200_decode_static(const sdpa_b200_params* p, void* stream) {
  using namespace sdpa_b200;
  // argument checks first, the device last: a refused request never needs a GPU
  int st = validate_forward_args(p);
  if (st != SDPA_B200_OK) return st;
  if (p->kernel == SDPA_B200_KERNEL_PREFILL) {
    set_error("decode_static runs the split-KV decode kernel only (kernel must be AUTO or DECODE)");
    return SDPA_B200_UNSUPPORTED;
  }
  st = check_decode_request(*p);
  if (st != SDPA_B200_OK) return st;
  DecodeParams d;
  plan_decode(*p, kPlanSms, d);
  const size_t need = partial_rows(*p, d) * sizeof(float) * (p->head_dim + 1);
  if (need > SDPA_B200_STATIC_SCRATCH_BYTES) {
    set_error("decode_static: batch %d x heads_q %d x %d splits needs %zu bytes of split partials, more than the "
              "%u bytes built into the library; lower num_splits or use sdpa_b200_fwd with a workspace",
              p->batch, p->heads_q, p->num_splits, need, static_cast<unsigned>(SDPA_B200_STATIC_SCRATCH_BYTES));
    return SDPA_B200_INVALID_ARG;
  }
  st = check_device();
  if (st != SDPA_B200_OK) return st;
  const int sms = sm_count();
  if (sms <= 0 || sms > kPlanSms) {
    set_error("decode_static: cannot use a device with %d SMs", sms);
    return SDPA_B200_NO_DEVICE;
  }
  void* scratch = nullptr;
  st = static_scratch_address(&scratch);
  if (st != SDPA_B200_OK) return st;
  plan_decode(*p, sms, d);
  uint32_t* status = p->device_status != nullptr ? p->device_status : static_cast<uint32_t*>(scratch);
  return launch_decode(*p, d, reinterpret_cast<float*>(static_cast<char*>(scratch) + kStaticHeaderBytes), status, "decode_static",
                       static_cast<cudaStream_t>(stream));
}
