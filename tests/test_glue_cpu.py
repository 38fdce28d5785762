"""The dispatcher glue without a GPU: it builds, loads, defines the four operators with the
reference's schemas and the backend toggles behave like the reference's."""
import re

import pytest
import torch

from torch_mlu_b200 import backends, ops, sdp_choice, torch_glue

# codegen/mlu_functions.yaml:1313-1316 of the reference
REFERENCE_SCHEMAS = {
    "_scaled_dot_product_flash_attention": "(Tensor query, Tensor key, Tensor value, float dropout_p=0.0, bool is_causal=False, bool return_debug_mask=False, *, float? scale=None) -> (Tensor ouput, Tensor logsumexp, Tensor cum_seq_q, Tensor cum_seq_k, int max_q, int max_k, Tensor philox_seed, Tensor philox_offset, Tensor debug_attn_mask)",
    "_scaled_dot_product_flash_attention_backward": "(Tensor grad_out, Tensor query, Tensor key, Tensor value, Tensor out, Tensor logsumexp, Tensor cum_seq_q, Tensor cum_seq_k, int max_q, int max_k, float dropout_p, bool is_causal, Tensor philox_seed, Tensor philox_offset, *, float? scale=None) -> (Tensor grad_query, Tensor grad_key, Tensor grad_value)",
    "_flash_attention_forward": "(Tensor query, Tensor key, Tensor value, Tensor cum_seq_q, Tensor cum_seq_k, int max_q, int max_k, float dropout_p, bool is_causal, bool return_debug_mask, *, float? scale=None) -> (Tensor output, Tensor softmax_logsumexp, Tensor philox_seed, Tensor philox_offset, Tensor debug_attn_mask)",
    "_flash_attention_backward": "(Tensor grad_out, Tensor query, Tensor key, Tensor value, Tensor out, Tensor logsumexp, Tensor cum_seq_q, Tensor cum_seq_k, int max_q, int max_k, float dropout_p, bool is_causal, Tensor philox_seed, Tensor philox_offset, *, float? scale=None) -> (Tensor, Tensor, Tensor)",
}


def _norm(s):
    return re.sub(r"=0\.0\b", "=0.", s).replace(" ", "")


def test_glue_defines_reference_schemas():
    torch_glue.load()
    for name, sig in REFERENCE_SCHEMAS.items():
        schema = str(getattr(torch.ops.b200_sdpa, name).default._schema)
        assert _norm(schema) == _norm(f"b200_sdpa::{name}{sig}"), schema
    assert torch.ops.b200_sdpa._launch_count() >= 0


def test_sdp_kernel_toggles_restore_state():
    before = (backends.flash_sdp_enabled(), backends.mem_efficient_sdp_enabled(), backends.math_sdp_enabled())
    with backends.sdp_kernel(enable_flash=True, enable_math=False, enable_mem_efficient=False):
        assert backends.flash_sdp_enabled() and not backends.math_sdp_enabled()
        assert not backends.mem_efficient_sdp_enabled()
    assert (backends.flash_sdp_enabled(), backends.mem_efficient_sdp_enabled(), backends.math_sdp_enabled()) == before
    assert int(backends.SDPBackend.FLASH_ATTENTION) == 1 and int(backends.SDPBackend.ERROR) == -1


def test_keys_without_heads_raise():
    """The check comes before the devices are looked at, and is not a division by the number of heads."""
    q, kv = torch.zeros(1, 8, 1, 128, dtype=torch.bfloat16), torch.zeros(1, 0, 64, 128, dtype=torch.bfloat16)
    for call in (ops.decode_attention, ops.gqa_prefill):
        with pytest.raises(RuntimeError, match="must divide"):
            call(q, kv, kv)


@pytest.mark.gpu
def test_packed_keys_without_heads_raise(cuda_device):
    q, kv = (torch.zeros(16, h, 128, dtype=torch.bfloat16, device=cuda_device) for h in (8, 0))
    cu = torch.tensor([0, 16], dtype=torch.int32, device=cuda_device)
    with pytest.raises(RuntimeError, match="must divide"):
        ops._flash_attention_forward(q, kv, kv, cu, cu, 16, 16, 0.0, False, False)


@pytest.fixture
def no_glue(monkeypatch):
    """As on a machine where the torch glue cannot be built: no compiler, no headers of torch."""
    def fail(*args, **kwargs):
        raise RuntimeError("building the torch glue failed")
    monkeypatch.setattr(torch_glue, "calls", None)
    monkeypatch.setattr(torch_glue, "_load_error", None, raising=False)
    monkeypatch.setattr(torch_glue, "build", fail)


def test_math_backend_needs_no_glue(no_glue):
    q = torch.randn(2, 4, 8, 64)
    with backends.sdp_kernel(enable_flash=True, enable_math=True, enable_mem_efficient=True):
        out = sdp_choice.scaled_dot_product_attention(q, q, q, is_causal=True)
    assert torch.allclose(out, torch.nn.functional.scaled_dot_product_attention(q, q, q, is_causal=True), atol=1e-5)


@pytest.mark.filterwarnings("ignore:the torch glue")
def test_ops_without_glue_check_their_arguments(no_glue, native_lib):
    q = torch.zeros(1, 8, 1, 128, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="must be on a CUDA device"):
        ops.decode_attention(q, q, q)
    with pytest.raises(RuntimeError, match="must divide"):
        ops.decode_attention(q, q[:, :0], q[:, :0])


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore:the torch glue")
def test_ops_without_glue_give_the_same_results(cuda_device, native_lib, monkeypatch, request):
    """The calls through ctypes are those of the native module: outputs, logsumexp and gradients bit for bit."""
    g = torch.Generator().manual_seed(1)
    q, k, v, do = (torch.randn(2, h, 200, 64, generator=g).bfloat16().to(cuda_device) for h in (8, 4, 4, 8))
    cu = torch.tensor([0, 150, 400], dtype=torch.int32, device=cuda_device)
    tq, tk, tv, tdo = (t.transpose(1, 2).flatten(0, 1) for t in (q, k, v, do))
    bias = torch.randn(1, 8, 200, 200, generator=g).bfloat16().to(cuda_device)

    def all_calls():
        out, lse = ops.gqa_prefill(q, k, v, is_causal=True)
        res = [out, lse, *ops._dense_backward(do, q, k, v, out, lse, True, 0.125, deterministic=True),
               *ops._dense_backward(do[:, :, :1].expand_as(do), q, k, v, out, lse, True, 0.125)]
        res += ops.decode_attention(q[:, :, :1], k, v)
        prepared = ops._prepare_bias(bias, q, k)
        out, lse = ops._dense_forward(q, k, v, False, None, True, bias=prepared)
        res += [out, lse, *ops._dense_backward(do, q, k, v, out, lse, False, 0.125, bias=prepared)]
        packed = ops._flash_attention_forward(tq, tk, tv, cu, cu, 250, 250, 0.0, True, False)
        res += [*packed, *ops._flash_attention_backward(tdo, tq, tk, tv, *packed[:2], cu, cu, 250, 250, 0.0, True, *packed[2:4])]
        assert ops.device_status() == 0
        return res

    want = all_calls()
    request.getfixturevalue("no_glue")
    monkeypatch.setattr(ops._Workspace, "_status", {})
    got = all_calls()
    assert torch_glue.calls is None and len(got) == len(want)
    for a, b in zip(got, want):
        assert torch.equal(a, b) and a.stride() == b.stride()
