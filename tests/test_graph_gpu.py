"""The C-ABI calls enqueue work on the caller's stream and nothing else (no allocation, no hidden
synchronisation), so forward + backward can be captured in a CUDA graph and replayed on new data."""
import pytest
import torch

from torch_mlu_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,D", [
    (2, 4, 128),
    (4, 26, 128),  # 312 forward units and 624 key blocks: the forward's unit counter, the dS GEMM and its unit counter
    (4, 26, 64),   # the fused backward and its accumulator's clearing
    (1, 2, 256),
])
def test_forward_backward_replay_in_a_cuda_graph(cuda_device, native_lib, B, H, D):
    dev = cuda_device
    g = torch.Generator().manual_seed(41)
    L = 768
    scale = D ** -0.5
    make = lambda: torch.randn(B, H, L, D, generator=g).bfloat16().to(dev)
    q, k, v, do = make(), make(), make(), make()
    side = torch.cuda.Stream(dev)
    side.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(side):  # warm-up outside capture: library handles, kernel attributes
        out, lse = ops.gqa_prefill(q, k, v, is_causal=True)
        ops._dense_backward(do, q, k, v, out, lse, True, scale)
    torch.cuda.current_stream(dev).wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, lse = ops.gqa_prefill(q, k, v, is_causal=True)
        dq, dk, dv = ops._dense_backward(do, q, k, v, out, lse, True, scale)
    for _ in range(2):  # replay twice on fresh inputs: the persistent kernel's unit counter is reset by a graph node too
        for t in (q, k, v, do):
            t.copy_(torch.randn(B, H, L, D, generator=g).bfloat16())
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in (out, lse, dq, dk, dv)]
        o2, l2 = ops.gqa_prefill(q, k, v, is_causal=True)
        want = [o2, l2, *ops._dense_backward(do, q, k, v, o2, l2, True, scale)]
        assert ops.device_status() == 0
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
            if name == "dq" and D == 64:
                # the fused kernel sums dQ in a varying order: two roundings to 16 bits of nearly the same sum
                assert float((a.float() - b.float()).norm() / b.float().norm()) <= 1e-3
            else:
                assert torch.equal(a, b), name


@pytest.mark.parametrize("call", ["prefill", "prefill_d256", "packed", "packed_d256", "decode", "decode_shared"])
@pytest.mark.parametrize("captured", [False, True])
def test_calls_launched_under_the_kernel_in_front_of_them(cuda_device, native_lib, call, captured):
    """Small forwards and decodes start under the tail of whatever is in front of them in the stream: they must see what that writes, and
    what follows must not touch their inputs early. The same calls with the device waited for between them give the same bits."""
    dev = cuda_device
    gen = torch.Generator(device=dev).manual_seed(5)
    randn = lambda *s: torch.randn(*s, generator=gen, device=dev, dtype=torch.bfloat16)
    call, D = call.replace("_d256", ""), 256 if call.endswith("d256") else 64
    B, H, Lq, Lk = {"prefill": (2, 4, 200, 200), "packed": (1, 4, 300, 300), "decode": (64, 8, 1, 64), "decode_shared": (2, 8, 1, 1500)}[call]
    shape = (lambda L: (L, H, D)) if call == "packed" else (lambda L: (B, H, L, D))
    src, q, k, v = randn(*shape(Lq)), randn(*shape(Lq)), randn(*shape(Lk)), randn(*shape(Lk))
    k0 = k.clone()
    cu = torch.tensor([0, 130, 300], dtype=torch.int32, device=dev)
    cu_written = torch.zeros_like(cu)

    def steps(wait):
        outs = []
        k.copy_(k0)
        for i in range(6):
            q.copy_(src)                   # a copy in front
            torch.mul(k, -1.0, out=k)      # a kernel in front
            cu_written.copy_(cu)
            wait()
            if call == "packed":
                out = ops._flash_attention_forward(q, k, v, cu_written, cu_written, 170, 170, 0.0, True, False)[0]
            else:
                out = ops.gqa_prefill(q, k, v, is_causal=True) if call == "prefill" else ops.decode_attention(q, k, v)
            outs.append(out if torch.is_tensor(out) else out[0])
            wait()
            q.zero_()                      # a kernel behind
            cu_written.zero_()
            k.add_(0.01)
        return outs

    want = [t.clone() for t in steps(torch.cuda.synchronize)]
    if captured:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = steps(lambda: None)
        for _ in range(3):
            g.replay()
    else:
        got = steps(lambda: None)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    for a, b in zip(got, want):
        assert torch.equal(a, b)
