"""The backward that leaves dS tiles in the workspace and takes dQ (head_dim 65 to 128, more key blocks than SMs), or dK and dQ
(head_dim above 128), from GEMMs over them."""
import ctypes

import pytest
import torch

from torch_mlu_b200 import _cabi, ops
from torch_mlu_b200.dropout import KeepMasks
from tests.test_guard_bands_gpu import set_bwd

pytestmark = pytest.mark.gpu
NAN = float("nan")


def run(lib, p, q, k, v, dout, packed, least):
    """dq, dk, dv through the C entry point, with a workspace full of NaN of the best or the least size."""
    grads = [torch.full_like(t, NAN) for t in (q, k, v)]
    set_bwd(p, dout, *grads, packed=packed)
    p.deterministic = 1  # both paths are; without it the least workspace has room for an accumulator, which may be as large as dS
    need, other = ctypes.c_size_t(0), ctypes.c_size_t(0)
    _cabi.check(lib.sdpa_b200_bwd_workspace_bytes(ctypes.byref(p), ctypes.byref(need)), "workspace query")
    _cabi.check(lib.sdpa_b200_bwd_workspace_least_bytes(ctypes.byref(p), ctypes.byref(other)), "workspace query")
    assert need.value > other.value, "this call does not take dS through the workspace"
    if least:
        need = other
    ws = torch.full(((need.value + 3) // 4,), NAN, device=q.device)
    stream = torch.cuda.current_stream(q.device).cuda_stream
    _cabi.check(lib.sdpa_b200_bwd(ctypes.byref(p), ws.data_ptr(), need.value, stream), "bwd")
    torch.cuda.synchronize()
    return grads


def gradients_in_64_bits(q, k, v, dout, causal):
    """[heads, length, head_dim] each."""
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    group = q.size(0) // k.size(0)
    s = q @ k.repeat_interleave(group, 0).transpose(1, 2) * q.size(-1) ** -0.5
    if causal:
        s = s.masked_fill(~torch.ones_like(s[0], dtype=torch.bool).tril(k.size(1) - q.size(1)), float("-inf"))
    out = torch.softmax(s, -1).nan_to_num(0.0) @ v.repeat_interleave(group, 0)
    return torch.autograd.grad(out, (q, k, v), dout.double())


def distance(got, want):
    return float((got.double() - want).norm() / want.norm())


def check(with_ds, without, want=None):
    # both sum the same products of 16-bit P and dS in the same order: where dS finds room is no matter of bits
    for i, name in enumerate(("dq", "dk", "dv")):
        assert torch.equal(with_ds[i], without[i]), name
        assert want is None or distance(with_ds[i], want[i]) < 4e-3, (name, distance(with_ds[i], want[i]))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,Hq,Hkv,Lq,Lk,D,causal", [
    (1, 60, 60, 257, 257, 128, True),     # one row in the third tile of queries and of keys
    (2, 28, 28, 257, 384, 128, True),     # mask offset 127
    (1, 80, 80, 384, 255, 72, True),      # more queries than keys: rows, and whole tiles of rows, that see nothing
    (1, 80, 80, 300, 129, 128, True),
    (1, 100, 50, 385, 385, 96, False),    # grouped queries, an odd number of 128-row tiles per unit pair
    (1, 160, 40, 130, 513, 128, False),
    (3, 60, 60, 128, 128, 128, True),     # one tile per head
    (1, 2, 2, 128, 192, 256, True),       # mask offset 64: a key block's first query block is hidden, its half of the tile zeros
    (2, 4, 2, 321, 513, 256, True),       # grouped; one row in the last query block
    (1, 3, 3, 400, 300, 136, True),       # queries that see nothing
    (2, 2, 1, 65, 257, 192, False),       # an odd number of key tiles
    (1, 1, 1, 1, 2, 256, False),
])
def test_dense(cuda_device, native_lib, B, Hq, Hkv, Lq, Lk, D, causal, dtype):
    gen = torch.Generator().manual_seed(5)
    q, k, v, dout = (torch.randn(B, h, n, D, generator=gen).to(cuda_device, dtype)
                     for h, n in ((Hq, Lq), (Hkv, Lk), (Hkv, Lk), (Hq, Lq)))
    out, lse = ops.gqa_prefill(q, k, v, is_causal=causal)
    p = ops._dense_params(q, k, v, out, lse, causal, D ** -0.5)
    want = [torch.stack(g) for g in zip(*(gradients_in_64_bits(q[b], k[b], v[b], dout[b], causal) for b in range(B)))]
    check(run(native_lib, p, q, k, v, dout, False, False), run(native_lib, p, q, k, v, dout, False, True), want)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lens_q,lens_k,Hq,Hkv,D", [
    ((257, 0, 1, 128, 130), (257, 5, 1, 128, 130), 40, 20, 128),
    ((100, 300, 129), (400, 300, 65), 60, 60, 128),   # shorter and longer keys than queries
    ((100, 0, 300, 129), (400, 7, 364, 65), 4, 2, 256),
])
def test_packed(cuda_device, native_lib, lens_q, lens_k, Hq, Hkv, D, causal):
    dev = cuda_device
    gen = torch.Generator().manual_seed(6)
    q, k, v, dout = (torch.randn(sum(n), h, D, generator=gen).to(dev, torch.bfloat16)
                     for n, h in ((lens_q, Hq), (lens_k, Hkv), (lens_k, Hkv), (lens_q, Hq)))
    ends_q, ends_k = ([sum(n[:i]) for i in range(len(n) + 1)] for n in (lens_q, lens_k))
    cu_q, cu_k = (torch.tensor(e, dtype=torch.int32, device=dev) for e in (ends_q, ends_k))
    args = (cu_q, cu_k, max(lens_q), max(lens_k), causal, D ** -0.5)
    out, lse = ops._varlen_forward(q, k, v, *args)
    p = ops._varlen_params(q, k, v, out, lse, *args)
    want = [torch.zeros_like(t, dtype=torch.float64) for t in (q, k, v)]
    for i, n in enumerate(lens_q):
        a, b = slice(ends_q[i], ends_q[i + 1]), slice(ends_k[i], ends_k[i + 1])
        if n > 0:
            one = gradients_in_64_bits(*(t.transpose(0, 1) for t in (q[a], k[b], v[b], dout[a])), causal)
            for w, g, rows in zip(want, one, (a, b, b)):
                w[rows] = g.transpose(0, 1)
    check(run(native_lib, p, q, k, v, dout, True, False), run(native_lib, p, q, k, v, dout, True, True), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,dropout,bias", [(128, True, None), (256, True, None), (80, False, "key"), (128, True, "key"),
                                            (128, False, "full"), (128, False, "full, not transposed"), (72, True, "full")])
def test_options(cuda_device, native_lib, D, dropout, bias, dtype):
    dev = cuda_device
    gen = torch.Generator(device=dev).manual_seed(9)
    B, H, Lq, Lk = 2, 28, 257, 392
    rand = lambda *shape: torch.randn(*shape, generator=gen, device=dev, dtype=dtype)
    q, k, v, dout = (rand(B, H, n, D) for n in (Lq, Lk, Lk, Lq))
    keep = KeepMasks(3, 4, 0.2, B, H, Lq, Lk, dev) if dropout else None
    b = bias_t = None
    if bias == "key":
        b = rand(B, 1, 1, Lk).expand(B, H, Lq, Lk)
    elif bias is not None:
        b = rand(1, H, Lq, Lk).expand(B, H, Lq, Lk)
        bias_t = ops._transposed_bias(b) if bias == "full" else None
    out, lse = ops._dense_forward(q, k, v, False, None, True, keep=keep, bias=b)
    p = ops._dense_params(q, k, v, out, lse, False, D ** -0.5)
    rows, cols, drop = (None, None, 0.0) if keep is None else (keep.rows, keep.cols, keep.dropout_p)
    ops._FieldCalls._options(p, rows, cols, drop, b, None, bias_t)
    want = None
    if not dropout:
        q64, k64, v64 = (t.double().requires_grad_() for t in (q, k, v))
        s = q64 @ k64.transpose(2, 3) * D ** -0.5 + b
        want = torch.autograd.grad(torch.softmax(s, -1) @ v64, (q64, k64, v64), dout.double())
    check(run(native_lib, p, q, k, v, dout, False, False), run(native_lib, p, q, k, v, dout, False, True), want)


@pytest.mark.parametrize("packed", [False, True])
def test_infinite_gradient_of_hidden_queries(cuda_device, native_lib, packed):
    """Keys from 128 on do not see queries 0 to 63, the first half of a dS tile: an infinite dO there leaves their gradients alone."""
    gen = torch.Generator().manual_seed(8)
    Lq, Lk, H, D = 128, 192, 3, 256
    q, k, v, dout = (torch.randn(1, H, n, D, generator=gen).to(cuda_device, torch.bfloat16) for n in (Lq, Lk, Lk, Lq))
    dout[0, :, 10] = float("inf")
    if packed:
        q, k, v, dout = (t[0].transpose(0, 1).contiguous() for t in (q, k, v, dout))
        cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device=cuda_device) for n in (Lq, Lk))
        args = (cu_q, cu_k, Lq, Lk, True, D ** -0.5)
        out, lse = ops._varlen_forward(q, k, v, *args)
        p = ops._varlen_params(q, k, v, out, lse, *args)
    else:
        out, lse = ops.gqa_prefill(q, k, v, is_causal=True)
        p = ops._dense_params(q, k, v, out, lse, True, D ** -0.5)
    for least in (False, True):
        dq, dk, dv = run(native_lib, p, q, k, v, dout, packed, least)
        if not packed:
            dq, dk, dv = (t[0].transpose(0, 1) for t in (dq, dk, dv))
        assert torch.isfinite(dk[128:]).all() and torch.isfinite(dv[128:]).all()
        assert torch.isfinite(torch.cat((dq[:10], dq[11:]))).all()


@pytest.mark.parametrize("native", [True, False])
def test_short_of_memory(cuda_device, native_lib, native):
    """178 MB of dS where torch may have 128 more: the same bits, and its pool, which empties its cache before it refuses, is asked once."""
    dev = cuda_device
    gen = torch.Generator(device=dev).manual_seed(10)
    q, k, v, dout = (torch.randn(1, 40, 2048, 128, generator=gen, device=dev, dtype=torch.bfloat16) for _ in range(4))
    out, lse = ops.gqa_prefill(q, k, v, is_causal=True)

    def backward():
        if native:
            return ops._dense_backward(dout, q, k, v, out, lse, True, 128 ** -0.5)
        grads = [torch.empty_like(t) for t in (q, k, v)]
        p = ops._dense_params(q, k, v, out, lse, True, 128 ** -0.5)
        set_bwd(p, dout, *grads, packed=False)
        ops._run_bwd(p, dev)
        return grads

    want = backward()
    ops._Workspace._bufs.clear()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    ooms = lambda: torch.cuda.memory_stats(dev)["num_ooms"]
    before = ooms()
    total = torch.cuda.get_device_properties(dev).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(dev) + (128 << 20)) / total, dev)
    try:
        for _ in range(3):
            for a, b in zip(backward(), want):
                assert torch.equal(a, b)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, dev)
    assert ooms() == before + 1
    # a thousand such calls later there is room, and it is used again
    for _ in range(1000 - 2 - 1):
        backward()
    torch.cuda.synchronize()
    for room in (False, True):
        torch.cuda.reset_peak_memory_stats(dev)
        used = torch.cuda.memory_allocated(dev)
        backward()
        assert (torch.cuda.max_memory_allocated(dev) - used > (178 << 20)) == room

def test_several_passes_over_the_workspace(cuda_device, native_lib):
    """2.7 GB of dS: two passes of ten heads give the bits of two calls with ten heads each."""
    gen = torch.Generator(device=cuda_device).manual_seed(7)
    q, k, v, dout = (torch.randn(1, 20, 8192, 128, generator=gen, device=cuda_device, dtype=torch.bfloat16) for _ in range(4))
    out, lse = ops.gqa_prefill(q, k, v, is_causal=False)
    whole = ops._dense_backward(dout, q, k, v, out, lse, False, 128 ** -0.5)
    for part in (slice(0, 10), slice(10, 20)):
        half = ops._dense_backward(*(t[:, part] for t in (dout, q, k, v, out)), lse[:, part].contiguous(), False, 128 ** -0.5)
        for a, b in zip(whole, half):
            assert torch.equal(a[:, part], b)


def test_the_backward_leaves_l2_to_the_kernels_behind_it(cuda_device, native_lib):
    """An addition over 48 + 48 MB, which fit L2, repeated behind a backward whose dS does not: from the third one on it takes what it takes behind a fill of the same
    size. Medians of 7 x 7 device times on either side, which differ by less than 1 % from run to run; dS lines that stay in L2 cost it 9 %."""
    from torch.profiler import ProfilerActivity, profile
    gen = torch.Generator(device=cuda_device).manual_seed(3)
    q, k, v, do = (torch.randn(4, 16, 2048, 128, generator=gen, device=cuda_device, dtype=torch.bfloat16) for _ in range(4))
    out, lse = ops.gqa_prefill(q, k, v, is_causal=True)
    big = torch.empty(280 << 20, device=cuda_device, dtype=torch.uint8)
    x, y = torch.zeros(12 << 20, device=cuda_device), torch.zeros(12 << 20, device=cuda_device)

    def behind(first):
        times = []
        for i in range(10):
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                first()
                for _ in range(9):
                    torch.add(x, 1.0, out=y)
                torch.cuda.synchronize()
            adds = sorted((e for e in prof.events() if "CUDAFunctor" in e.name and "add" in e.name.lower()), key=lambda e: e.time_range.start)
            if i >= 3:
                times += [e.device_time for e in adds[2:]]
        assert len(times) >= 35  # the profiler may lose some
        return sorted(times)[len(times) // 2]

    backward = behind(lambda: ops._dense_backward(do, q, k, v, out, lse, True, 128 ** -0.5))
    fill = behind(lambda: big.fill_(1))
    assert backward <= 1.04 * fill, (backward, fill)
