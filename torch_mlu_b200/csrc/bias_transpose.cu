// Preparation of attention biases: a boolean mask as a bias (mask_to_bias_kernel), a bias with rows of a multiple of 8 keys
// (bias_pad_kernel), its gradient summed over what it is broadcast along (bias_grad_sum_kernel), and the transposed copy for the backward
// pass: [.., Lq, Lk] -> [.., Lk, ld >= Lq].
//
// The dK/dV kernel's threads own keys and walk over queries, so it reads a bias stored query-major two bytes
// at a time; with this copy (sdpa_b200_params.bias_t) it reads 16 bytes at a time. HBM-bound: every element is
// read once and written once through a 64 x 64 shared-memory tile, 16 bytes per thread on both sides.
#include "kernels.h"
#include "ptx_sm100.cuh"

namespace sdpa_b200 {
namespace {

struct TransposeParams {
  const uint16_t* src;
  uint16_t* dst;
  int64_t batch_stride, head_stride, row_stride;  // of src, in elements
  int heads, seqlen_q, seqlen_k, ld;
};

__global__ void __launch_bounds__(256) bias_transpose_kernel(const TransposeParams p) {
  // [key][query]; 33 words per row: the transposing 2-byte writes of a warp (rows 8 apart) fall on 4 banks instead of
  // one, the 4-byte reads of the second phase on 32 different banks
  __shared__ uint16_t tile[64][66];
  const int t = threadIdx.x;
  const int q0 = blockIdx.y * 64, k0 = blockIdx.x * 64;
  const int z = blockIdx.z, b = z / p.heads, h = z - b * p.heads;
  const uint16_t* src = p.src + b * p.batch_stride + h * p.head_stride;
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    const int r = pass * 32 + (t >> 3), c = (t & 7) * 8;
    const int q = q0 + r, k = k0 + c;
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    // a chunk that straddles the last key reads row padding, which the bias rules guarantee
    if (q < p.seqlen_q && k < p.seqlen_k) w = *reinterpret_cast<const uint4*>(src + static_cast<int64_t>(q) * p.row_stride + k);
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint16_t e = static_cast<uint16_t>(ww[i >> 1] >> ((i & 1) * 16));
      tile[c + i][r] = (k + i < p.seqlen_k) ? e : static_cast<uint16_t>(0);
    }
  }
  __syncthreads();
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    const int kr = pass * 32 + (t >> 3), c = (t & 7) * 8;
    const int k = k0 + kr, q = q0 + c;
    if (k < p.seqlen_k && q < p.ld) {
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[i] = static_cast<uint32_t>(tile[kr][c + 2 * i]) | (static_cast<uint32_t>(tile[kr][c + 2 * i + 1]) << 16);
      *reinterpret_cast<uint4*>(p.dst + (static_cast<int64_t>(z) * p.seqlen_k + k) * p.ld + q) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// Boolean mask -> 0 / -inf bias, eight keys (16 bytes of output) per thread. Launch-bound for the usual padding masks (a few
// KB); one kernel where the tensor-library route took three (fill, invert, masked fill) and a copy for unaligned rows.
struct MaskParams {
  const uint8_t* mask;
  uint4* out;
  int64_t batch_stride, head_stride, row_stride, key_stride;
  int heads, seqlen_q, seqlen_k, groups;  // groups: 8-key groups per output row
  uint32_t neg_inf;                       // -inf in both halves
};

__global__ void __launch_bounds__(256) mask_to_bias_kernel(const MaskParams p, int64_t total) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int64_t row = i / p.groups;
  const int k0 = static_cast<int>(i - row * p.groups) * 8;
  const int64_t bh = row / p.seqlen_q;
  const int64_t b = bh / p.heads;
  const uint8_t* src = p.mask + b * p.batch_stride + (bh - b * p.heads) * p.head_stride + (row - bh * p.seqlen_q) * p.row_stride;
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int k = k0 + 2 * j;
    uint32_t x = 0u;
    if (k < p.seqlen_k && src[k * p.key_stride] == 0) x |= p.neg_inf & 0x0000ffffu;
    if (k + 1 < p.seqlen_k && src[(k + 1) * p.key_stride] == 0) x |= p.neg_inf & 0xffff0000u;
    w[j] = x;
  }
  p.out[i] = make_uint4(w[0], w[1], w[2], w[3]);
}

// The same for a bias in its own type, whose rows the attention kernels cannot read where they lie: bound by memory, one launch where filling and copying took
// two and wrote the copy twice (12 heads of 594 x 594 11.9 us -> 6.7, 192 of 1001 x 1001 524 -> 216).
struct PadParams {
  const uint16_t* bias;
  uint4* out;
  int64_t batch_stride, head_stride, row_stride, key_stride;
  int heads, seqlen_q, seqlen_k, groups;
};
__global__ void __launch_bounds__(256) bias_pad_kernel(const PadParams p, int64_t total) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int64_t row = i / p.groups;
  const int k0 = static_cast<int>(i - row * p.groups) * 8;
  const int64_t bh = row / p.seqlen_q;
  const int64_t b = bh / p.heads;
  const uint16_t* src = p.bias + b * p.batch_stride + (bh - b * p.heads) * p.head_stride + (row - bh * p.seqlen_q) * p.row_stride;
  uint32_t v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = k0 + j < p.seqlen_k ? src[(k0 + j) * p.key_stride] : 0u;
  p.out[i] = make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16), v[4] | (v[5] << 16), v[6] | (v[7] << 16));
}

// Sums a [batch, heads, seqlen_q, seqlen_k] gradient over batches and / or heads, eight keys per thread, fp32. Bound by memory and, behind it, by instructions: eight
// reads are in flight per thread, addresses are counted on instead of divided out. (Behind the kernel that writes the gradient, tensor library's sum | one thread per
// element | so: 16 batches of 12 heads of 594 x 594, 135 MB, 52 us | 42 | 38; 2 of 8 of 2000 x 2000 114 | 85 | 72; 40 of 12 of 384 x 384 36 | 47 | 47, with
// 128-byte reads per thread too short for its many streams.) Where the result is small, `slices` threads share an element's summands, every slices-th eight of them, and
// their sums meet in shared memory, in the order of the threads: in one thread, the 512 summands of a [64, 64] bias of B32 H16 are 64 memory latencies one behind the
// other on two SMs (16 | 163 | 8; [197, 197] of B16 H12 20 | 65 | 6.6; 256 batches of 8 heads of 100 x 100 14.6 | 106 | 15.8).
struct GradSumParams {
  const uint16_t* grad;
  uint16_t* out;  // contiguous
  int64_t batch_stride, head_stride, row_stride;
  int out_heads, sum_batches, sum_heads;  // heads of the result; batches and heads per element of it
  int seqlen_q, seqlen_k, groups;
  int slices;       // a power of two up to kSumThreads / 8
  bool wide_rows;   // rows of the result are whole groups at 16-byte addresses
};
constexpr int kSumThreads = 256;
template <bool kF16>
__global__ void __launch_bounds__(kSumThreads) bias_grad_sum_kernel(const GradSumParams p, int64_t total) {
  __shared__ float4 sums[2][kSumThreads];
  const int elements = kSumThreads / p.slices;  // groups of eight keys per block
  const int slice = threadIdx.x / elements;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * elements + (threadIdx.x - slice * elements);
  int64_t row, b;
  int h, q, k0;
  if (total <= 0xffffffffll) {  // divisions of 64 bits take as long as the loads
    const uint32_t r = static_cast<uint32_t>(i) / p.groups, bh = r / p.seqlen_q;
    k0 = static_cast<int>(static_cast<uint32_t>(i) - r * p.groups) * 8;
    q = static_cast<int>(r - bh * p.seqlen_q);
    row = r;
    b = bh / p.out_heads;
    h = static_cast<int>(bh - static_cast<uint32_t>(b) * p.out_heads);
  } else {
    row = i / p.groups;
    k0 = static_cast<int>(i - row * p.groups) * 8;
    const int64_t bh = row / p.seqlen_q;
    q = static_cast<int>(row - bh * p.seqlen_q);
    b = bh / p.out_heads;
    h = static_cast<int>(bh - b * p.out_heads);
  }
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (i < total) {
    const uint16_t* src = p.grad + b * p.batch_stride + h * p.head_stride + q * p.row_stride + k0;
    const int n = p.sum_batches * p.sum_heads;
    const int64_t next_batch = p.batch_stride - static_cast<int64_t>(p.sum_heads - 1) * p.head_stride;
    for (int first = slice * 8; first < n; first += p.slices * 8) {
      const int sb = first / p.sum_heads;
      int sh = first - sb * p.sum_heads;
      const uint16_t* at = src + sb * p.batch_stride + sh * p.head_stride;
      uint4 w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        w[u] = first + u < n ? __ldg(reinterpret_cast<const uint4*>(at)) : make_uint4(0u, 0u, 0u, 0u);
        const bool last = ++sh == p.sum_heads;
        at += last ? next_batch : p.head_stride;
        sh = last ? 0 : sh;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint32_t ww[4] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 x = unpack_16x2<kF16>(ww[j]);
          acc[2 * j] += x.x;
          acc[2 * j + 1] += x.y;
        }
      }
    }
  }
  if (p.slices > 1) {
    sums[0][threadIdx.x] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    sums[1][threadIdx.x] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    __syncthreads();
    if (slice != 0) return;
    for (int other = threadIdx.x + elements; other < kSumThreads; other += elements) {
      const float4 x = sums[0][other], y = sums[1][other];
      acc[0] += x.x;
      acc[1] += x.y;
      acc[2] += x.z;
      acc[3] += x.w;
      acc[4] += y.x;
      acc[5] += y.y;
      acc[6] += y.z;
      acc[7] += y.w;
    }
  }
  if (i >= total) return;
  uint16_t* dst = p.out + row * p.seqlen_k + k0;
  if (p.wide_rows) {
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_16x2<kF16>(acc[0], acc[1]), pack_16x2<kF16>(acc[2], acc[3]), pack_16x2<kF16>(acc[4], acc[5]),
                                                pack_16x2<kF16>(acc[6], acc[7]));
    return;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (k0 + j < p.seqlen_k) dst[j] = to_16<kF16>(acc[j]);
}

}  // namespace
}  // namespace sdpa_b200

using namespace sdpa_b200;

extern "C" SDPA_B200_API int sdpa_b200_mask_to_bias(const void* mask, int64_t batch_stride, int64_t head_stride, int64_t row_stride,
                                                    int64_t key_stride, int32_t batch, int32_t heads, int32_t seqlen_q,
                                                    int32_t seqlen_k, void* out, int64_t out_row_stride, int32_t dtype,
                                                    void* stream) {
  if (mask == nullptr || out == nullptr || (reinterpret_cast<uintptr_t>(out) & 15u) || batch <= 0 || heads <= 0 || seqlen_q <= 0 ||
      seqlen_k <= 0 || batch_stride < 0 || head_stride < 0 || row_stride < 0 || key_stride < 0 || (out_row_stride % 8) != 0 ||
      out_row_stride < seqlen_k || (dtype != SDPA_B200_BF16 && dtype != SDPA_B200_F16)) {
    set_error("mask_to_bias: non-NULL pointers, a 16-byte aligned output, positive sizes, strides that are not negative and "
              "an output row stride that is a multiple of 8 and holds seqlen_k");
    return SDPA_B200_INVALID_ARG;
  }
  MaskParams m;
  m.mask = static_cast<const uint8_t*>(mask);
  m.out = static_cast<uint4*>(out);
  m.batch_stride = batch_stride;
  m.head_stride = head_stride;
  m.row_stride = row_stride;
  m.key_stride = key_stride;
  m.heads = heads;
  m.seqlen_q = seqlen_q;
  m.seqlen_k = seqlen_k;
  m.groups = static_cast<int>(out_row_stride / 8);
  m.neg_inf = dtype == SDPA_B200_F16 ? 0xfc00fc00u : 0xff80ff80u;
  const int64_t total = static_cast<int64_t>(batch) * heads * seqlen_q * m.groups;
  const int64_t blocks = (total + 255) / 256;
  if (blocks > 0x7fffffff) {
    set_error("mask_to_bias: too many elements");
    return SDPA_B200_INVALID_ARG;
  }
  mask_to_bias_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(m, total);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("mask_to_bias: launch failed: %s", cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  return SDPA_B200_OK;
}

extern "C" SDPA_B200_API int sdpa_b200_transpose_bias(const void* bias, int64_t batch_stride, int64_t head_stride,
                                                      int64_t row_stride, int32_t batch, int32_t heads, int32_t seqlen_q,
                                                      int32_t seqlen_k, void* out, int64_t out_row_stride, void* stream) {
  auto bad = [](int64_t s) { return s < 0 || (s % 8) != 0; };
  if (bias == nullptr || out == nullptr || (reinterpret_cast<uintptr_t>(bias) & 15u) || (reinterpret_cast<uintptr_t>(out) & 15u) ||
      bad(batch_stride) || bad(head_stride) || bad(row_stride) || row_stride == 0) {
    set_error("transpose_bias: 16-byte aligned pointers, strides that are multiples of 8 elements and a non-zero row stride");
    return SDPA_B200_INVALID_ARG;
  }
  if (batch <= 0 || heads <= 0 || seqlen_q <= 0 || seqlen_k <= 0 || static_cast<int64_t>(batch) * heads > 65535 ||
      out_row_stride < (static_cast<int64_t>(seqlen_q) + 7) / 8 * 8 || (out_row_stride % 8) != 0) {
    set_error("transpose_bias: sizes must be positive, batch*heads at most 65535, out_row_stride a multiple of 8 that "
              "holds seqlen_q");
    return SDPA_B200_INVALID_ARG;
  }
  TransposeParams t;
  t.src = static_cast<const uint16_t*>(bias);
  t.dst = static_cast<uint16_t*>(out);
  t.batch_stride = batch_stride;
  t.head_stride = head_stride;
  t.row_stride = row_stride;
  t.heads = heads;
  t.seqlen_q = seqlen_q;
  t.seqlen_k = seqlen_k;
  t.ld = static_cast<int>(out_row_stride);
  dim3 grid((seqlen_k + 63) / 64, (static_cast<int>(out_row_stride) + 63) / 64, batch * heads);
  if (grid.y > 65535) {
    set_error("transpose_bias: seqlen_q too long (%d)", seqlen_q);
    return SDPA_B200_INVALID_ARG;
  }
  bias_transpose_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(t);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("transpose_bias: launch failed: %s", cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  return SDPA_B200_OK;
}

extern "C" SDPA_B200_API int sdpa_b200_pad_bias(const void* bias, int64_t batch_stride, int64_t head_stride, int64_t row_stride, int64_t key_stride,
                                                int32_t batch, int32_t heads, int32_t seqlen_q, int32_t seqlen_k, void* out,
                                                int64_t out_row_stride, void* stream) {
  if (bias == nullptr || out == nullptr || (reinterpret_cast<uintptr_t>(bias) & 1u) || (reinterpret_cast<uintptr_t>(out) & 15u) || batch <= 0 ||
      heads <= 0 || seqlen_q <= 0 || seqlen_k <= 0 || batch_stride < 0 || head_stride < 0 || row_stride < 0 || key_stride < 0 ||
      (out_row_stride % 8) != 0 || out_row_stride < seqlen_k) {
    set_error("pad_bias: non-NULL pointers, a 16-byte aligned output, positive sizes, strides that are not negative and an output row stride that is a "
              "multiple of 8 and holds seqlen_k");
    return SDPA_B200_INVALID_ARG;
  }
  PadParams m;
  m.bias = static_cast<const uint16_t*>(bias);
  m.out = static_cast<uint4*>(out);
  m.batch_stride = batch_stride;
  m.head_stride = head_stride;
  m.row_stride = row_stride;
  m.key_stride = key_stride;
  m.heads = heads;
  m.seqlen_q = seqlen_q;
  m.seqlen_k = seqlen_k;
  m.groups = static_cast<int>(out_row_stride / 8);
  const int64_t total = static_cast<int64_t>(batch) * heads * seqlen_q * m.groups, blocks = (total + 255) / 256;
  if (blocks > 0x7fffffff) {
    set_error("pad_bias: too many elements");
    return SDPA_B200_INVALID_ARG;
  }
  bias_pad_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(m, total);
  const cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("pad_bias: launch failed: %s", cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  return SDPA_B200_OK;
}

extern "C" SDPA_B200_API int sdpa_b200_sum_bias_grad(const void* grad, int64_t batch_stride, int64_t head_stride, int64_t row_stride, int32_t batch,
                                                     int32_t heads, int32_t seqlen_q, int32_t seqlen_k, int32_t over_batch, int32_t over_heads,
                                                     void* out, int32_t dtype, void* stream) {
  auto bad = [](int64_t s) { return s < 0 || (s % 8) != 0; };
  if (grad == nullptr || out == nullptr || (reinterpret_cast<uintptr_t>(grad) & 15u) || (reinterpret_cast<uintptr_t>(out) & 1u) || batch <= 0 ||
      heads <= 0 || seqlen_q <= 0 || seqlen_k <= 0 || bad(batch_stride) || bad(head_stride) || bad(row_stride) || row_stride < seqlen_k ||
      (dtype != SDPA_B200_BF16 && dtype != SDPA_B200_F16)) {
    set_error("sum_bias_grad: non-NULL pointers, a 16-byte aligned gradient, positive sizes and strides that are multiples of 8, with rows that are readable "
              "to the next multiple of 8 keys");
    return SDPA_B200_INVALID_ARG;
  }
  GradSumParams m;
  m.grad = static_cast<const uint16_t*>(grad);
  m.out = static_cast<uint16_t*>(out);
  m.batch_stride = batch_stride;
  m.head_stride = head_stride;
  m.row_stride = row_stride;
  m.out_heads = over_heads ? 1 : heads;
  m.sum_batches = over_batch ? batch : 1;
  m.sum_heads = over_heads ? heads : 1;
  m.seqlen_q = seqlen_q;
  m.seqlen_k = seqlen_k;
  m.groups = (seqlen_k + 7) / 8;
  const int64_t total = static_cast<int64_t>(over_batch ? 1 : batch) * m.out_heads * seqlen_q * m.groups;
  m.wide_rows = seqlen_k % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  // until every thread has one eight of summands, or the SMs the threads that they hold: beyond, a thread costs more than its shorter chain gives (figures above)
  m.slices = 1;
  while (m.slices < kSumThreads / 8 && total * m.slices < 148 * 2048 && static_cast<int64_t>(m.sum_batches) * m.sum_heads > 8 * m.slices) m.slices *= 2;
  const int per_block = kSumThreads / m.slices;
  const int64_t blocks = (total + per_block - 1) / per_block;
  if (blocks > 0x7fffffff) {
    set_error("sum_bias_grad: too many elements");
    return SDPA_B200_INVALID_ARG;
  }
  auto kernel = dtype == SDPA_B200_F16 ? bias_grad_sum_kernel<true> : bias_grad_sum_kernel<false>;
  kernel<<<static_cast<unsigned>(blocks), kSumThreads, 0, static_cast<cudaStream_t>(stream)>>>(m, total);
  const cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) {
    set_error("sum_bias_grad: launch failed: %s", cudaGetErrorString(err));
    return SDPA_B200_LAUNCH_FAILED;
  }
  count_launch();
  return SDPA_B200_OK;
}
