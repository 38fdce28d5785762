// Interface between the parts of the torch glue: torch_glue.cpp (argument checks, parameter blocks, the dispatcher
// operators), sdpa_autograd.cpp (autograd formulas, the scaled_dot_product_attention front end) and py_calls.cpp (the
// direct Python entry points behind ops.py and sdp_choice.py).
#pragma once

#include <ATen/ATen.h>

#include <string>
#include <tuple>

#include "../../include/sdpa_b200.h"

namespace b200_glue {

// A C-ABI call returned a non-zero status (the Python entry points turn it into _cabi.SdpaError).
class StatusError : public c10::Error {
 public:
  StatusError(int status, std::string text) : c10::Error({__func__, __FILE__, static_cast<uint32_t>(__LINE__)}, std::move(text)), status_(status) {}
  int status() const { return status_; }

 private:
  int status_;
};

inline void check_status(int st, const char* what) {
  if (C10_LIKELY(st == SDPA_B200_OK)) return;
  throw StatusError(st, c10::str(what, ": ", sdpa_b200_status_string(st), ": ", sdpa_b200_last_error()));
}

// One bit per (query, key) pair in both orientations, written by the library from a Philox seed / offset pair
// (the reference draws the pattern inside its kernel from such a pair and hands the pair to the backward
// operator, FlashAttention_internal.cpp:190-214).
struct KeepMasks {
  at::Tensor rows, cols;  // int32 [B*H, Lq_pad, Lk_pad/32] and [B*H, Lk_pad, Lq_pad/32]
  double p = 0.0;
};

struct ForwardOptions {
  int kernel = SDPA_B200_KERNEL_AUTO;
  int num_splits = 0;
  int sm_margin = 0;
  const KeepMasks* keep = nullptr;
  const at::Tensor* bias = nullptr;  // [B, H, Lq, Lk] view from prepare_bias()
};

struct BackwardOptions {
  const KeepMasks* keep = nullptr;
  const at::Tensor* bias = nullptr;
  const at::Tensor* dbias = nullptr;   // zero-filled, rows padded to a multiple of 8
  const at::Tensor* bias_t = nullptr;  // the bias with keys and queries exchanged
  int deterministic = -1;              // 1 / 0; -1: torch.are_deterministic_algorithms_enabled()
};

double scale_or_default(const at::Tensor& q, c10::optional<double> scale);

// One int32 per device that every call made through this glue hands to the kernels.
at::Tensor& status_word(int device);

std::tuple<at::Tensor, at::Tensor> dense_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, bool causal,
                                                 double scale, bool allow_gqa, const ForwardOptions& opt = {});
std::tuple<at::Tensor, at::Tensor, at::Tensor> dense_backward(const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k,
                                                              const at::Tensor& v, const at::Tensor& out, const at::Tensor& lse,
                                                              bool causal, double scale, const BackwardOptions& opt = {});
std::tuple<at::Tensor, at::Tensor> varlen_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                                  const at::Tensor& cu_q, const at::Tensor& cu_k, int64_t max_q, int64_t max_k,
                                                  bool causal, double scale, const ForwardOptions& opt = {});
std::tuple<at::Tensor, at::Tensor, at::Tensor> varlen_backward(const at::Tensor& dout, const at::Tensor& q, const at::Tensor& k,
                                                               const at::Tensor& v, const at::Tensor& out, const at::Tensor& lse,
                                                               const at::Tensor& cu_q, const at::Tensor& cu_k, int64_t max_q,
                                                               int64_t max_k, bool causal, double scale,
                                                               const BackwardOptions& opt = {});

// The operator pairs with dropout_p: seed / offset are CPU int64 scalars, or empty device tensors when dropout_p is 0.
struct DropoutResult {
  at::Tensor out, lse, seed, offset, debug;
};
DropoutResult dense_forward_with_dropout(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, double dropout_p,
                                         bool causal, bool return_debug_mask, double scale, bool allow_gqa);
std::tuple<at::Tensor, at::Tensor, at::Tensor> dense_backward_with_dropout(
    const at::Tensor& grad_out, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& out,
    const at::Tensor& lse, double dropout_p, bool causal, const at::Tensor& philox_seed, const at::Tensor& philox_offset,
    double scale);
DropoutResult varlen_forward_with_dropout(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& cu_q,
                                          const at::Tensor& cu_k, int64_t max_q, int64_t max_k, double dropout_p, bool causal,
                                          double scale, bool return_debug_mask = false);
std::tuple<at::Tensor, at::Tensor, at::Tensor> varlen_backward_with_dropout(
    const at::Tensor& grad_out, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& out,
    const at::Tensor& lse, const at::Tensor& cu_q, const at::Tensor& cu_k, int64_t max_q, int64_t max_k, double dropout_p,
    bool causal, const at::Tensor& philox_seed, const at::Tensor& philox_offset, double scale);

// sdpa_autograd.cpp: scaled_dot_product_attention on the fused kernels, with autograd. An undefined tensor when the call
// is not one of the plain cases served here (the caller then goes through the full choice procedure of sdp_choice.py).
at::Tensor sdpa(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const c10::optional<at::Tensor>& attn_mask,
                double dropout_p, bool is_causal, c10::optional<double> scale);

}  // namespace b200_glue
