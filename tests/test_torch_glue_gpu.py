"""The dispatcher glue on a GPU: the b200_sdpa operators (reference schemas) with autograd, and
the opt-in aten overrides that put F.scaled_dot_product_attention on these kernels."""
import pytest
import torch
import torch.nn.functional as F

from oracle import sdpa_oracle as orc
from torch_mlu_b200 import _cabi, backends, torch_glue

pytestmark = pytest.mark.gpu


def rand(shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(shape, generator=g).bfloat16()


def test_registered_ops_forward_backward_autograd(cuda_device, native_lib):
    torch_glue.load()
    dev = cuda_device
    q, k, v, do = (rand((2, 4, 384, 128), s) for s in (1, 2, 3, 4))
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    res = torch.ops.b200_sdpa._scaled_dot_product_flash_attention(qd, kd, vd, 0.0, True, False)
    out, lse = res[0], res[1]
    assert len(res) == 9 and res[4] == 384 and res[5] == 384
    out.backward(do.to(dev))
    o_ref, l_ref = orc.cpu_sdpa_forward(q, k, v, causal=True)
    dq, dk, dv = orc.cpu_sdpa_backward(do, q, k, v, o_ref, l_ref, causal=True)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_lse(lse, l_ref)
    orc.assert_close_grad_bf16(qd.grad, dq, "dq")
    orc.assert_close_grad_bf16(kd.grad, dk, "dk")
    orc.assert_close_grad_bf16(vd.grad, dv, "dv")


def test_registered_varlen_op_autograd(cuda_device, native_lib):
    torch_glue.load()
    dev = cuda_device
    lens = [100, 260, 33]
    cu = [0, 100, 360, 393]
    q, k, v, do = rand((393, 4, 128), 1), rand((393, 2, 128), 2), rand((393, 2, 128), 3), rand((393, 4, 128), 4)
    cu_t = torch.tensor(cu, dtype=torch.int32, device=dev)
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    out, lse, *_ = torch.ops.b200_sdpa._flash_attention_forward(qd, kd, vd, cu_t, cu_t, max(lens), max(lens), 0.0, True, False)
    out.backward(do.to(dev))
    o_ref, l_ref = orc.varlen_forward(q, k, v, cu, cu, causal=True)
    dq, dk, dv = orc.varlen_backward(do, q, k, v, cu, cu, causal=True)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_lse(lse, l_ref)
    orc.assert_close_grad_bf16(qd.grad, dq, "dq")
    orc.assert_close_grad_bf16(kd.grad, dk, "dk")
    orc.assert_close_grad_bf16(vd.grad, dv, "dv")


def test_functional_sdpa_reaches_these_kernels_when_overridden(cuda_device, native_lib):
    """Same call pattern as the reference tests: F.scaled_dot_product_attention inside
    sdp_kernel(enable_flash=True, enable_math=False, enable_mem_efficient=False)
    (test/torch_ops/test_scaled_dot_product_attention.py:630-640)."""
    dev = cuda_device
    q, k, v, do = (rand((1, 16, 512, 128), s) for s in (1, 2, 3, 4))
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    torch_glue.install_aten_overrides()
    try:
        before = _cabi.launch_count()
        with backends.sdp_kernel(enable_flash=True, enable_math=False, enable_mem_efficient=False):
            out = F.scaled_dot_product_attention(qd, kd, vd, is_causal=True)
        out.backward(do.to(dev))
        torch.cuda.synchronize()
        assert _cabi.launch_count() - before == 4  # forward + (preprocess, dK/dV, dQ)
    finally:
        torch_glue.remove_aten_overrides()
    o_ref, l_ref = orc.cpu_sdpa_forward(q, k, v, causal=True)
    dq, dk, dv = orc.cpu_sdpa_backward(do, q, k, v, o_ref, l_ref, causal=True)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_grad_bf16(qd.grad, dq, "dq")
    orc.assert_close_grad_bf16(kd.grad, dk, "dk")
    orc.assert_close_grad_bf16(vd.grad, dv, "dv")
    # with the overrides removed the stock kernel is back (no launches of this library)
    before = _cabi.launch_count()
    with backends.sdp_kernel(enable_flash=True, enable_math=False, enable_mem_efficient=False):
        F.scaled_dot_product_attention(qd.detach(), kd.detach(), vd.detach(), is_causal=True)
    torch.cuda.synchronize()
    assert _cabi.launch_count() == before


def test_glue_rejects_what_the_reference_rejects(cuda_device, native_lib):
    torch_glue.load()
    dev = cuda_device
    q = rand((1, 2, 64, 128), 1).to(dev)
    with pytest.raises(RuntimeError, match="same number of heads"):
        torch.ops.b200_sdpa._scaled_dot_product_flash_attention(q, q[:, :1], q[:, :1])
    with pytest.raises(RuntimeError, match="fp16 and bf16"):
        torch.ops.b200_sdpa._scaled_dot_product_flash_attention(q.float(), q.float(), q.float())
    with pytest.raises(RuntimeError, match="dropout_p must be inside"):
        torch.ops.b200_sdpa._scaled_dot_product_flash_attention(q, q, q, 1.0)
    wide = torch.cat([q, q, q[..., :64]], dim=-1)  # head_dim 320: beyond what the reference admits (sdp_utils.h:231-255)
    with pytest.raises(RuntimeError, match="at most 256"):
        torch.ops.b200_sdpa._scaled_dot_product_flash_attention(wide, wide, wide)


@pytest.mark.parametrize("amp_dtype", [torch.bfloat16, torch.float16])
def test_autocast_casts_fp32_inputs_like_the_reference(cuda_device, native_lib, amp_dtype):
    """aten/autocast_mode.cpp:147 puts _scaled_dot_product_flash_attention on the
    lower_precision_fp list: fp32 inputs run in the autocast dtype, gradients come back in fp32."""
    torch_glue.load()
    dev = cuda_device
    g = torch.Generator().manual_seed(11)
    q, k, v, do = (torch.randn((1, 2, 256, 128), generator=g) for _ in range(4))
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    with torch.autocast("cuda", dtype=amp_dtype):
        out = torch.ops.b200_sdpa._scaled_dot_product_flash_attention(qd, kd, vd, 0.0, True, False)[0]
    assert out.dtype == amp_dtype
    out.backward(do.to(dev).to(amp_dtype))
    assert qd.grad.dtype == torch.float32
    ql, kl, vl, dl = (t.to(amp_dtype) for t in (q, k, v, do))
    o_ref, l_ref = orc.cpu_sdpa_forward(ql, kl, vl, causal=True)
    dq, dk, dv = orc.cpu_sdpa_backward(dl, ql, kl, vl, o_ref, l_ref, causal=True)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_grad_bf16(qd.grad, dq, "dq")
    orc.assert_close_grad_bf16(kd.grad, dk, "dk")
    orc.assert_close_grad_bf16(vd.grad, dv, "dv")


def _attention_with_mask(q, k, v, keep, p, causal, dtype=torch.float32):
    qf, kf, vf = (t.to(dtype).detach().requires_grad_(True) for t in (q, k, v))
    scores = torch.einsum("bhtd,bhsd->bhts", qf * (q.shape[-1] ** -0.5), kf)
    if causal:
        scores = scores.masked_fill(orc.causal_mask_bottom_right(q.shape[2], k.shape[2]), float("-inf"))
    attn = torch.softmax(scores, dim=-1).masked_fill(~keep, 0.0) / (1.0 - p)
    return torch.einsum("bhts,bhsd->bhtd", attn, vf), (qf, kf, vf)


def test_dropout_through_the_registered_operator_and_autograd(cuda_device, native_lib):
    """dropout_p > 0 with return_debug_mask, as the reference tests call it (test_...py:1018-1026): the operator
    returns the pattern and the Philox pair; autograd's backward replays the pattern from the pair."""
    torch_glue.load()
    dev = cuda_device
    p = 0.22
    q, k, v = (rand((2, 3, 260, 128), s) for s in (1, 2, 3))
    do = torch.rand((2, 3, 260, 128), generator=torch.Generator().manual_seed(4)).bfloat16()
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    res = torch.ops.b200_sdpa._scaled_dot_product_flash_attention(qd, kd, vd, p, True, True)
    out, seed, offset, debug = res[0], res[6], res[7], res[8]
    assert seed.numel() == 1 and offset.numel() == 1 and tuple(debug.shape) == (2, 3, 260, 260)
    keep = (debug > 0).cpu()
    visible = ~orc.causal_mask_bottom_right(260, 260)
    assert torch.equal(keep & visible, orc.dropout_keep_mask(int(seed), int(offset), p, 2, 3, 260, 260) & visible)
    out.backward(do.to(dev))
    ref, (qf, kf, vf) = _attention_with_mask(q, k, v, keep, p, True)
    ref.backward(do.float())
    lp, (ql, kl, vl) = _attention_with_mask(q, k, v, keep, p, True, torch.bfloat16)
    lp.backward(do)
    orc.assert_close_bf16(out, ref.detach(), "out")
    orc.assert_close_reference_rule(qd.grad, qf.grad, ql.grad, "dq", fudge=4)
    orc.assert_close_reference_rule(kd.grad, kf.grad, kl.grad, "dk")
    orc.assert_close_reference_rule(vd.grad, vf.grad, vl.grad, "dv")


def test_functional_sdpa_with_dropout_uses_the_cuda_generator(cuda_device, native_lib):
    """F.scaled_dot_product_attention(dropout_p=...) on the overridden aten operators: the pattern comes from the
    device generator's (seed, offset), which the test reads before the call to rebuild the expected result."""
    dev = cuda_device
    p = 0.3
    q, k, v = (rand((1, 4, 256, 128), s) for s in (1, 2, 3))
    do = torch.rand((1, 4, 256, 128), generator=torch.Generator().manual_seed(4)).bfloat16()
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    torch_glue.install_aten_overrides()
    try:
        torch.cuda.manual_seed(4242)
        gen = torch.cuda.default_generators[dev.index or 0]
        seed, offset = gen.initial_seed(), gen.get_offset()
        with backends.sdp_kernel(enable_flash=True, enable_math=False, enable_mem_efficient=False):
            out = F.scaled_dot_product_attention(qd, kd, vd, dropout_p=p, is_causal=True)
            again = F.scaled_dot_product_attention(qd, kd, vd, dropout_p=p, is_causal=True)
        out.backward(do.to(dev))
    finally:
        torch_glue.remove_aten_overrides()
    assert not torch.equal(out, again)          # the generator moved on
    keep = orc.dropout_keep_mask(seed, offset, p, 1, 4, 256, 256)
    ref, (qf, kf, vf) = _attention_with_mask(q, k, v, keep, p, True)
    ref.backward(do.float())
    orc.assert_close_bf16(out, ref.detach(), "out")
    orc.assert_close_grad_bf16(qd.grad, qf.grad, "dq")
    orc.assert_close_grad_bf16(kd.grad, kf.grad, "dk")
    orc.assert_close_grad_bf16(vd.grad, vf.grad, "dv")


def test_packed_operator_with_dropout_and_autograd(cuda_device, native_lib):
    """b200_sdpa::_flash_attention_forward with dropout_p > 0: the Philox pair comes back, autograd's backward
    replays the pattern, and everything matches fp32 math with the pattern rebuilt on the CPU."""
    torch_glue.load()
    dev = cuda_device
    p, H, D = 0.22, 2, 128
    lens = [130, 257]
    cu = [0, 130, 387]
    q, k, v = (rand((387, H, D), s) for s in (1, 2, 3))
    do = torch.rand((387, H, D), generator=torch.Generator().manual_seed(4)).bfloat16()
    cu_t = torch.tensor(cu, dtype=torch.int32, device=dev)
    qd, kd, vd = (t.to(dev).requires_grad_(True) for t in (q, k, v))
    out, lse, seed, offset, _ = torch.ops.b200_sdpa._flash_attention_forward(qd, kd, vd, cu_t, cu_t, 257, 257, p, True, False)
    assert seed.numel() == 1 and offset.numel() == 1
    out.backward(do.to(dev))
    for b, L in enumerate(lens):
        sl = slice(cu[b], cu[b + 1])
        one = lambda x: x[sl].transpose(0, 1).unsqueeze(0)
        keep = orc.dropout_keep_mask(int(seed), int(offset), p, len(lens), H, L, L)[b:b + 1]
        ref, (qf, kf, vf) = _attention_with_mask(one(q), one(k), one(v), keep, p, True)
        ref.backward(one(do).float())
        orc.assert_close_bf16(one(out), ref.detach(), f"out[{b}]")
        orc.assert_close_grad_bf16(one(qd.grad), qf.grad, f"dq[{b}]")
        orc.assert_close_grad_bf16(one(kd.grad), kf.grad, f"dk[{b}]")
        orc.assert_close_grad_bf16(one(vd.grad), vf.grad, f"dv[{b}]")


@pytest.mark.parametrize("which", ["query", "value", "mask"])
@pytest.mark.parametrize("requires_grad", [False, True])
def test_forward_mode_raises(cuda_device, native_lib, which, requires_grad):
    """A tangent is not dropped in silence, by the package's function or by the registered operators."""
    import torch.autograd.forward_ad as fwd
    dev = cuda_device
    q, k, v = (torch.randn(2, 4, 128, 64, device=dev, dtype=torch.bfloat16, requires_grad=requires_grad) for _ in range(3))
    bias = torch.randn(1, 4, 128, 128, device=dev, dtype=torch.bfloat16)
    cu = torch.tensor([0, 128], dtype=torch.int32, device=dev)
    from torch_mlu_b200 import sdp_choice
    with fwd.dual_level():
        dual = lambda t: fwd.make_dual(t, torch.ones_like(t))
        if which == "query":
            q = dual(q)
        elif which == "value":
            v = dual(v)
        with pytest.raises(NotImplementedError):
            sdp_choice.scaled_dot_product_attention(q, k, v, attn_mask=dual(bias) if which == "mask" else bias)
        if which != "mask":
            with pytest.raises(NotImplementedError):
                sdp_choice.scaled_dot_product_attention(q, k, v)
            with pytest.raises(NotImplementedError):
                torch.ops.b200_sdpa._scaled_dot_product_flash_attention(q, k, v)
            with pytest.raises(NotImplementedError):
                torch.ops.b200_sdpa._flash_attention_forward(q[0].transpose(0, 1), k[0].transpose(0, 1), v[0].transpose(0, 1), cu, cu,
                                                             128, 128, 0.0, False, False)


def _qkv_and_bias(dev, requires_grad=False):
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(2, 4, 128, 64, generator=g).bfloat16().to(dev).requires_grad_(requires_grad) for _ in range(3))
    return q, k, v, torch.randn(1, 4, 128, 128, generator=g).bfloat16().to(dev)


class _Logged(torch.Tensor):
    seen = []

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.seen.append(getattr(func, "__name__", str(func)))
        return super().__torch_function__(func, types, args, kwargs or {})


class _FunctionLog(torch.overrides.TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


def test_package_function_is_seen_by_torch_function(cuda_device, native_lib):
    """Subclasses and modes with __torch_function__ see the attention operator, and a subclass comes back as one."""
    from torch_mlu_b200 import sdp_choice
    q, k, v, _ = _qkv_and_bias(cuda_device)
    want = sdp_choice.scaled_dot_product_attention(q, k, v)
    out = sdp_choice.scaled_dot_product_attention(q.as_subclass(_Logged), k, v)
    assert type(out) is _Logged and "_scaled_dot_product_flash_attention" in _Logged.seen and torch.equal(out.as_subclass(torch.Tensor), want)
    with _FunctionLog() as log:
        assert torch.equal(sdp_choice.scaled_dot_product_attention(q, k, v), want)
    assert any("_scaled_dot_product_flash_attention" in f for f in log.seen)


@pytest.mark.parametrize("masked", [False, True])
def test_package_function_under_transforms_and_tracing(cuda_device, native_lib, masked):
    """Wrapped tensors do not reach the kernels: what has no rule for them raises, as the operators do, or gives the same result."""
    from torch_mlu_b200 import sdp_choice
    q, k, v, bias = _qkv_and_bias(cuda_device)
    mask = bias if masked else None
    f = lambda q, k, v: sdp_choice.scaled_dot_product_attention(q, k, v, attn_mask=mask)
    want = f(q, k, v)
    if masked:
        with pytest.raises(RuntimeError, match="setup_context"):
            torch.func.functionalize(f)(q, k, v)
        traced = torch.jit.trace(f, (q, k, v), check_trace=False)
        q2 = torch.flip(q, [0])
        assert torch.equal(traced(q2, k, v), f(q2, k, v))
    else:
        assert torch.equal(torch.func.functionalize(f)(q, k, v), want)
        with pytest.raises(RuntimeError, match="[Bb]atching rule"):
            torch.func.vmap(f)(*(torch.stack([t, t]) for t in (q, k, v)))
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.jvp(lambda q: f(q, k, v), (q,), (torch.ones_like(q),))
    with pytest.raises(RuntimeError, match="torch.func|functorch"):
        torch.func.grad(lambda q: f(q, k, v).float().sum())(q)
    qg = q.clone().requires_grad_()
    assert f(qg, k, v).requires_grad
    if not masked:
        with torch._C._AutoDispatchBelowAutograd():
            assert not f(qg, k, v).requires_grad
    neg = torch._neg_view(q)  # a lazily negated view of q: its memory holds q, not -q
    assert torch.equal(f(neg, k, v), f(-q, k, v)) or masked


class _DispatchLog(torch.utils._python_dispatch.TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


def _call(form, q, k, v, bias, dropout_p=0.0):
    """The package's function or a registered operator on the same values; `form` also names the backward operator's suffix."""
    from torch_mlu_b200 import sdp_choice
    if form == "packed":
        cu = torch.arange(q.size(0) + 1, device=q.device, dtype=torch.int32) * q.size(2)
        tokens = [t.transpose(1, 2).flatten(0, 1) for t in (q, k, v)]
        return torch.ops.b200_sdpa._flash_attention_forward(*tokens, cu, cu, q.size(2), q.size(2), dropout_p, False, False)[0]
    return sdp_choice.scaled_dot_product_attention(q, k, v, attn_mask=bias if form == "bias" else None, dropout_p=dropout_p)


BACKWARD_OPS = {"dense": "b200_sdpa._scaled_dot_product_flash_attention_backward.default",
                "packed": "b200_sdpa._flash_attention_backward.default", "bias": "b200_sdpa._bias_attention_backward.default"}


@pytest.mark.parametrize("form", ["dense", "packed", "bias"])
def test_dispatch_modes_see_the_backward(cuda_device, native_lib, form):
    q, k, v, bias = _qkv_and_bias(cuda_device, requires_grad=True)
    bias.requires_grad_()
    inputs = (q, k, v, bias) if form == "bias" else (q, k, v)
    out = _call(form, q, k, v, bias)
    go = torch.randn_like(out)
    want = torch.autograd.grad(out, inputs, go, retain_graph=True)
    with _DispatchLog() as log:
        got = torch.autograd.grad(out, inputs, go)
    assert BACKWARD_OPS[form] in log.seen, log.seen
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("dropout_p", [0.0, 0.1])
@pytest.mark.parametrize("form", ["dense", "packed"])
def test_make_fx_records_the_backward(cuda_device, native_lib, form, dropout_p):
    """The traced program computes the gradients of the inputs it is given, not those of the tracing call."""
    from torch.fx.experimental.proxy_tensor import make_fx
    q, k, v, _ = _qkv_and_bias(cuda_device, requires_grad=True)

    def step(q, k, v):
        out = _call(form, q, k, v, None, dropout_p)
        return torch.autograd.grad(out, (q, k, v), torch.ones_like(out))

    traced = make_fx(step)(q, k, v)
    assert BACKWARD_OPS[form] in [str(n.target) for n in traced.graph.nodes]
    if dropout_p == 0.0:
        q2, k2, v2 = (torch.flip(t.detach(), [0]).requires_grad_() for t in (q, k, v))
        for a, b in zip(traced(q2, k2, v2), step(q2, k2, v2)):
            assert torch.equal(a, b)


def test_batched_gradients(cuda_device, native_lib):
    q, k, v, _ = _qkv_and_bias(cuda_device, requires_grad=True)
    out = _call("dense", q, k, v, None)
    go = torch.randn(2, *out.shape, device=cuda_device, dtype=out.dtype)
    got = torch.autograd.grad(out, (q, k, v), go, is_grads_batched=True, retain_graph=True)
    for i in range(2):
        for a, b in zip(got, torch.autograd.grad(out, (q, k, v), go[i], retain_graph=True)):
            assert torch.equal(a[i], b)


@pytest.mark.parametrize("dropout_p", [0.0, 0.1])
@pytest.mark.parametrize("form", ["dense", "packed", "bias", "mask"])
def test_compiled_autograd(cuda_device, native_lib, form, dropout_p):
    """The recorded backward, run again on other values, gives what the eager one does."""
    from torch._dynamo import compiled_autograd
    from torch_mlu_b200 import sdp_choice
    if dropout_p > 0.0 and form in ("bias", "mask"):
        pytest.skip("dropout with an attn_mask has its own Python autograd function")
    torch._dynamo.reset()
    graphs = []

    def grads(seed, compiled):
        q, k, v, bias = (torch.flip(t, [0]) if seed else t.clone() for t in _qkv_and_bias(cuda_device))
        inputs = [t.requires_grad_() for t in ((q, k, v, bias) if form == "bias" else (q, k, v))]
        torch.cuda.manual_seed(seed)
        if form == "mask":
            out = sdp_choice.scaled_dot_product_attention(q, k, v, attn_mask=bias > -1)
        else:
            out = _call(form, q, k, v, bias, dropout_p)
        if compiled:
            with compiled_autograd._enable(lambda gm: (graphs.append(gm), gm)[1]):
                out.float().sum().backward()
        else:
            out.float().sum().backward()
        return [t.grad for t in inputs]

    for seed in (0, 1):
        for a, b in zip(grads(seed, True), grads(seed, False)):
            assert torch.equal(a, b)
    names = [str(n.target) for gm in graphs for n in gm.graph.nodes]
    assert any("B200AttentionBackward" in n for n in names), names


@pytest.mark.parametrize("view", ["expanded_rows", "expanded_all", "one_row", "odd_rows", "unaligned", "columns"])
@pytest.mark.parametrize("form,D", [("dense", 64), ("dense", 256), ("packed", 128), ("bias", 64)])
def test_gradients_of_any_layout(cuda_device, native_lib, form, D, view):
    """What autograd hands back for sums, slices of concatenations and transposed consumers gives the gradients of its copy."""
    B, H, L = 2, 4, 1 if view == "one_row" else 96
    g = torch.Generator().manual_seed(2)
    q, k, v = (torch.randn(B, H, L, D, generator=g).bfloat16().to(cuda_device).requires_grad_() for _ in range(3))
    bias = torch.randn(1, H, L, L, generator=g).bfloat16().to(cuda_device)
    out = _call(form, q, k, v, bias)
    shape = out.shape
    rows = 0 if form == "packed" else 2
    if view in ("expanded_rows", "one_row"):
        go = torch.randn([1 if i == rows else n for i, n in enumerate(shape)], generator=g).bfloat16().to(cuda_device).expand(shape)
        go = go.as_strided(shape, [0 if i == rows else s for i, s in enumerate(go.stride())])
    elif view == "expanded_all":
        go = torch.randn([], generator=g).bfloat16().to(cuda_device).expand(shape)
    elif view == "odd_rows":
        go = torch.randn(*shape[:-1], D + 3, generator=g).bfloat16().to(cuda_device)[..., :D]
    elif view == "unaligned":
        go = torch.randn(*shape[:-1], D + 8, generator=g).bfloat16().to(cuda_device)[..., 1:D + 1]
    else:
        go = torch.randn(*shape[:-2], D, shape[-2], generator=g).bfloat16().to(cuda_device).transpose(-1, -2)
    want = torch.autograd.grad(out, (q, k, v), go.clone(memory_format=torch.contiguous_format), retain_graph=True)
    for a, b in zip(torch.autograd.grad(out, (q, k, v), go), want):
        assert torch.equal(a, b)


def test_outputs_are_filled_under_deterministic_algorithms(cuda_device, native_lib):
    """torch fills memory that an operator leaves unwritten: here the rows of tokens that belong to no sequence."""
    from torch_mlu_b200 import ops
    q = torch.randn(300, 4, 64, device=cuda_device).bfloat16()
    cu = torch.tensor([0, 100, 200], dtype=torch.int32, device=cuda_device)
    torch.use_deterministic_algorithms(True)
    try:
        out, lse = ops._flash_attention_forward(q, q, q, cu, cu, 100, 100, 0.0, False, False)[:2]
    finally:
        torch.use_deterministic_algorithms(False)
    assert out[200:].isnan().all() and lse[:, 200:].isnan().all() and not out[:200].isnan().any()
