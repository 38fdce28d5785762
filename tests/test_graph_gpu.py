"""The C-ABI calls enqueue work on the caller's stream and nothing else (no allocation, no hidden
synchronisation), so forward + backward can be captured in a CUDA graph and replayed on new data."""
import pytest
import torch

from torch_mlu_b200 import _cabi, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,D,L", [
    (2, 4, 128, 768),
    (4, 26, 128, 768),  # 312 forward units, taken from waiting CTAs, and 624 key blocks: the dS GEMM and its unit counter
    (4, 26, 64, 768),   # the dK/dV and the dQ kernel
    (2, 20, 64, 1100),  # the fused backward and its accumulator's clearing
    (1, 2, 256, 768),
])
def test_forward_backward_replay_in_a_cuda_graph(cuda_device, native_lib, B, H, D, L):
    dev = cuda_device
    g = torch.Generator().manual_seed(41)
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
    for _ in range(2):  # replay twice on fresh inputs
        for t in (q, k, v, do):
            t.copy_(torch.randn(B, H, L, D, generator=g).bfloat16())
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in (out, lse, dq, dk, dv)]
        o2, l2 = ops.gqa_prefill(q, k, v, is_causal=True)
        want = [o2, l2, *ops._dense_backward(do, q, k, v, o2, l2, True, scale)]
        assert ops.device_status() == 0
        for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
            if name == "dq" and D == 64 and L > 1024:
                # the fused kernel sums dQ in a varying order: two roundings to 16 bits of nearly the same sum
                assert float((a.float() - b.float()).norm() / b.float().norm()) <= 1e-3
            else:
                assert torch.equal(a, b), name


@pytest.mark.parametrize("call", ["prefill", "prefill_d256", "packed", "packed_d256", "decode", "decode_shared"])
@pytest.mark.parametrize("captured", [False, True])
def test_calls_launched_under_the_kernel_in_front_of_them(cuda_device, native_lib, call, captured):
    """Small forwards and decodes may start under the tail of whatever is in front of them in the stream (torch's kernels and copies here, which
    let nothing start early; captured calls do not overlap either): they must see what that writes, and
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
            q.copy_(src)                   # copies in front
            cu_written.copy_(cu)
            torch.mul(k, -1.0, out=k)      # and a kernel directly in front
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


@pytest.mark.parametrize("chain", ["prefill_64", "prefill_96_keys", "prefill_256", "packed_64", "packed_256", "counted_128", "decode_merge", "decode_merge_64",
                                   "decode_cluster", "decode_whole", "prefill_and_decode"])
def test_chains_of_calls_that_feed_one_another(cuda_device, native_lib, chain):
    """Calls of this library directly behind one another let the next one start before they have ended. Here each one's output is an input of the next, with
    nothing between them, and partial results of consecutive decodes share one piece of workspace: the bits are those of the same calls with the
    device waited for after each."""
    dev = cuda_device
    gen = torch.Generator(device=dev).manual_seed(6)
    randn = lambda *s: torch.randn(*s, generator=gen, device=dev).bfloat16()
    launches = None
    if chain.startswith("prefill_") and chain != "prefill_and_decode":
        D = int(chain.split("_")[1])
        x0, k, v = randn(2, 6, 200, D), randn(2, 6, 200, D), randn(2, 6, 200, D)
        step = (lambda x: ops.gqa_prefill(k, x, v, is_causal=True)[0]) if chain.endswith("keys") else (lambda x: ops.gqa_prefill(x, k, v, is_causal=True)[0])
        launches = 1
    elif chain.startswith("packed"):
        D = int(chain.split("_")[1])
        x0, k, v = randn(300, 4, D), randn(300, 4, D), randn(300, 4, D)
        cu = torch.tensor([0, 130, 300], dtype=torch.int32, device=dev)
        step = lambda x: ops._flash_attention_forward(x, k, x, cu, cu, 170, 170, 0.0, True, False)[0]
        launches = 1
    elif chain == "counted_128":  # more units than SMs, taken from waiting CTAs
        x0, k, v = randn(2, 80, 300, 128), randn(2, 80, 300, 128), randn(2, 80, 300, 128)
        step = lambda x: ops.gqa_prefill(x, k, v, is_causal=True)[0]
    elif chain == "prefill_and_decode":  # a forward's output is the decode's cache, the decode's output the forward's first query
        x0, q, k, v = randn(2, 8, 1, 128), randn(2, 8, 300, 128), randn(2, 8, 300, 128), randn(2, 8, 300, 128)

        def step(x):
            cache = ops.gqa_prefill(x.expand(2, 8, 1, 128), k, v, is_causal=False)[0]
            full = ops.gqa_prefill(q, k, v, is_causal=True)[0]
            return ops.decode_attention(cache, full, full)[0]
    else:
        B, Hq, Hkv, Lk, D, launches = {"decode_merge": (1, 8, 2, 4096, 128, 2), "decode_merge_64": (1, 40, 1, 9000, 64, 2),
                                       "decode_cluster": (1, 32, 8, 1000, 128, 1), "decode_whole": (30, 8, 8, 200, 64, 1)}[chain]
        x0, k, v = randn(B, Hq, 1, D), randn(B, Hkv, Lk, D), randn(B, Hkv, Lk, D)
        step = lambda x: ops.decode_attention(x, k, v)[0]

    def run(wait):
        x, outs = x0, []
        for _ in range(12):
            x = step(x)
            wait()
            outs.append(x)
        return outs

    before = _cabi.launch_count()
    want = run(torch.cuda.synchronize)
    if launches is not None:
        assert _cabi.launch_count() - before == 12 * launches
    for _ in range(3):
        got = run(lambda: None)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        for i, (a, b) in enumerate(zip(got, want)):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("B,H,D,L,causal", [(4, 26, 128, 768, True), (5, 32, 64, 256, False)])
def test_units_by_the_counter_replay_in_a_cuda_graph(cuda_device, native_lib, B, H, D, L, causal):
    """A call that leaves an SM free takes its units off the counter, whose clearing is a graph node too: two replays on new inputs, against the bits of the call
    that takes them from waiting CTAs or has none to leave."""
    dev = cuda_device
    gen = torch.Generator(device=dev).manual_seed(43)
    make = lambda: torch.randn(B, H, L, D, generator=gen, device=dev, dtype=torch.bfloat16)
    q, k, v = make(), make(), make()
    call = lambda margin: ops.gqa_prefill(q, k, v, is_causal=causal, sm_margin=margin)
    side = torch.cuda.Stream(dev)
    side.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(side):
        call(1)
    torch.cuda.current_stream(dev).wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, lse = call(1)
    for _ in range(2):
        for t in (q, k, v):
            t.copy_(make())
        graph.replay()
        torch.cuda.synchronize()
        want = call(0)
        assert ops.device_status() == 0
        assert torch.equal(out, want[0]) and torch.equal(lse, want[1])


def test_chain_of_calls_by_the_counter(cuda_device, native_lib):
    """The counter's clearing stands between calls of which each one's output is the next one's query: the bits are those of the same calls with the device waited for."""
    gen = torch.Generator(device=cuda_device).manual_seed(7)
    x0, k, v = (torch.randn(2, 80, 300, 128, generator=gen, device=cuda_device, dtype=torch.bfloat16) for _ in range(3))

    def run(wait, margin):
        x, outs = x0, []
        for _ in range(12):
            x = ops.gqa_prefill(x, k, v, is_causal=True, sm_margin=margin)[0]
            wait()
            outs.append(x)
        return outs

    want = run(torch.cuda.synchronize, 0)
    for _ in range(3):
        got = run(lambda: None, 1)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        for i, (a, b) in enumerate(zip(got, want)):
            assert torch.equal(a, b), i
