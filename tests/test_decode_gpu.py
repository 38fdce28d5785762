"""GPU parity of the split-KV decode kernel against the CPU oracle, through the C ABI."""
import pytest
import torch

from oracle import sdpa_oracle as orc
from torch_mlu_b200 import _cabi, ops, workloads

pytestmark = pytest.mark.gpu


def rand(shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(shape, generator=g).bfloat16()


@pytest.mark.parametrize("B,Hq,Hkv,Lk,splits", [
    (2, 8, 2, 1000, 1),
    (2, 8, 2, 1000, 4),
    (1, 4, 4, 4096, 0),
    (2, 32, 2, 777, 3),     # 16 query heads per KV head: both fragment row halves
    (1, 40, 1, 2048, 2),    # 40:1 MQA, three head chunks
    (3, 8, 8, 1, 1),        # single key
    (1, 8, 2, 63, 5),       # more splits than 64-key steps: empty splits
    (1, 32, 8, 8192, 0),
])
def test_decode_matches_oracle(cuda_device, native_lib, B, Hq, Hkv, Lk, splits):
    q, k, v = rand((B, Hq, 1, 128), 1), rand((B, Hkv, Lk, 128), 2), rand((B, Hkv, Lk, 128), 3)
    dev = cuda_device
    out, lse = ops.decode_attention(q.to(dev), k.to(dev), v.to(dev), num_splits=splits)
    o_ref, l_ref = orc.cpu_sdpa_forward(q, k, v, causal=False)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_lse(lse, l_ref)


@pytest.mark.parametrize("B,Hq,Hkv,Lk,D,launches", [
    (1, 8, 1, 20000, 128, 2),    # one unit over every CTA of the grid
    (5, 24, 1, 130, 64, 1),      # head chunks of 16 and 8, a tile of two keys: as clusters of two
    (1, 24, 1, 20000, 64, 2),    # head chunks of 16 and 8 in equal shares
    (1, 40, 2, 8192, 128, 2),    # of 16 and 4
    (7, 32, 2, 9000, 128, 2),    # 16 heads: a full chunk
    (75, 8, 4, 64, 128, 1),      # one tile per unit, more units than CTAs: nothing is shared
    (50, 8, 8, 65, 64, 2),       # 400 units of two tiles: shares that begin and end inside units
    (37, 12, 12, 700, 128, 2),   # 444 units: CTAs with whole units between two shared ones
])
def test_decode_equal_shares(cuda_device, native_lib, B, Hq, Hkv, Lk, D, launches):
    """The automatic split deals 64-key tiles of all (batch, kv head) units out in equal contiguous shares: shapes whose
    shares begin, end or lie entirely inside units. Two launches tell that shares were merged. Tolerances as above (16-bit output, fp32 logsumexp)."""
    q, k, v = rand((B, Hq, 1, D), 1), rand((B, Hkv, Lk, D), 2), rand((B, Hkv, Lk, D), 3)
    dev = cuda_device
    before = _cabi.launch_count()
    out, lse = ops.decode_attention(q.to(dev), k.to(dev), v.to(dev))
    assert ops.device_status() == 0 and _cabi.launch_count() - before == launches
    o_ref, l_ref = orc.cpu_sdpa_forward(q, k, v, causal=False)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_lse(lse, l_ref)


@pytest.mark.parametrize("B,Hq,Hkv,Lk,D,launches", [
    (1, 32, 8, 1000, 128, 1),   # clusters of 8, two tiles each, the last one short
    (1, 5, 1, 600, 64, 1),      # clusters of 8 that merge 20 column pairs each: part of a warp
    (1, 20, 2, 321, 64, 1),     # clusters of 4 over six tiles: the last CTA has none; ten heads: both fragment row halves
    (2, 40, 1, 600, 128, 1),    # the same with head chunks of 16, 16 and 8
    (12, 12, 12, 100, 128, 1),  # clusters of 2
    (1, 32, 8, 5000, 128, 2),   # too long for a cluster
    (30, 8, 8, 200, 64, 1),     # a nearly full wave of whole units
    (19, 8, 8, 130, 128, 2),    # half a wave of them
    (60, 16, 8, 130, 64, 1),    # two waves of whole units
    (68, 16, 16, 100, 64, 2),   # four waves of two tiles
    (35, 8, 8, 4097, 64, 1),    # several waves of clusters, 33 and 32 tiles each
    (30, 4, 4, 8129, 128, 1),   # nearly two waves of clusters of four
    (30, 4, 4, 8129, 64, 2),    # too few bytes in a share for them
    (9, 8, 8, 16385, 64, 2),    # not in waves of clusters of eight: equal shares
])
def test_decode_without_a_merge_kernel(cuda_device, native_lib, B, Hq, Hkv, Lk, D, launches):
    """Each side of the rule that chooses whole units, clusters or equal shares. Tolerances as above; the kernels are counted so that
    every case is on the side that it stands for."""
    q, k, v = rand((B, Hq, 1, D), 1), rand((B, Hkv, Lk, D), 2), rand((B, Hkv, Lk, D), 3)
    dev = cuda_device
    before = _cabi.launch_count()
    out, lse = ops.decode_attention(q.to(dev), k.to(dev), v.to(dev))
    assert ops.device_status() == 0 and _cabi.launch_count() - before == launches
    o_ref, l_ref = orc.cpu_sdpa_forward(q, k, v, causal=False)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_lse(lse, l_ref)


@pytest.mark.parametrize("what", ["query", "key", "value", "score"])
@pytest.mark.parametrize("B,Hq,Hkv,Lk,splits,D", [
    (1, 8, 2, 4096, 0, 128),    # every unit shared between CTAs
    (1, 40, 2, 1000, 0, 64),    # clusters of eight, head chunks of 16 and 4
    (1, 40, 2, 8192, 0, 128),   # equal shares, the same chunks
    (1, 24, 2, 20000, 0, 64),   # of 12 heads
    (1, 8, 2, 4096, 4, 128),    # fixed splits
    (1, 8, 2, 200, 6, 64),      # fixed splits, some of them without keys
    (2, 8, 2, 4096, 1, 128),    # one CTA per unit
    (160, 8, 2, 64, 0, 128),    # whole units
])
def test_decode_shows_nan_and_overflow(cuda_device, native_lib, B, Hq, Hkv, Lk, splits, D, what):
    """One NaN in an input, or one score that overflows to +inf, makes the rows that see it NaN however the keys are dealt
    out, as the softmax of the same values does; the other rows are not touched."""
    q, k, v = rand((B, Hq, 1, D), 1), rand((B, Hkv, Lk, D), 2), rand((B, Hkv, Lk, D), 3)
    at = 7 if Lk < 1000 else 300  # a key in the first share, the others hold none
    if what == "query":
        q[0, 1, 0, 5] = float("nan")
    elif what == "key":
        k[0, 1, at, 5] = float("nan")
    elif what == "value":
        v[0, 1, at, 5] = float("nan")
    else:
        q[0, :, 0, 0] = 0.0  # the other heads' scores stay ordinary
        q[0, 1, 0, 0] = k[0, 0, at, 0] = 1e20
    s = torch.einsum("bhqd,bhkd->bhqk", q.float(), k.float().repeat_interleave(Hq // Hkv, 1)) * D ** -0.5
    want = torch.einsum("bhqk,bhkd->bhqd", torch.softmax(s, -1), v.float().repeat_interleave(Hq // Hkv, 1))
    bad = want.isnan()
    assert bad.any() and not bad.all()
    dev = cuda_device
    out, lse = ops.decode_attention(q.to(dev), k.to(dev), v.to(dev), num_splits=splits)
    assert ops.device_status() == 0
    out = out.float().cpu()
    assert torch.equal(out.isnan(), bad)
    orc.assert_close_bf16(out.masked_fill(bad, 0.0).bfloat16(), want.masked_fill(bad, 0.0), "out")
    assert torch.equal(lse.cpu().isfinite(), ~s.softmax(-1).isnan().any(-1))


@pytest.mark.parametrize("B,Hq,Hkv,Lk,splits", [(2, 8, 2, 1000, 4), (1, 32, 2, 777, 3), (1, 4, 4, 4096, 0)])
def test_decode_head_dim_64(cuda_device, native_lib, B, Hq, Hkv, Lk, splits):
    g = torch.Generator().manual_seed(8)
    q = torch.randn((B, Hq, 1, 64), generator=g).bfloat16()
    k = torch.randn((B, Hkv, Lk, 64), generator=g).bfloat16()
    v = torch.randn((B, Hkv, Lk, 64), generator=g).bfloat16()
    dev = cuda_device
    out, lse = ops.decode_attention(q.to(dev), k.to(dev), v.to(dev), num_splits=splits)
    o_ref, l_ref = orc.cpu_sdpa_forward(q, k, v, causal=False)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_lse(lse, l_ref)


def test_decode_auto_dispatch_and_strided_cache(cuda_device, native_lib):
    """Lq == 1 reaches the decode kernel through the dense op too; the cache may be a
    [B, L, H, D] buffer viewed as [B, H, L, D]."""
    dev = cuda_device
    B, Hq, Hkv, Lk = 2, 8, 2, 1500
    q = rand((B, Hq, 1, 128), 1)
    kc = rand((B, Lk, Hkv, 128), 2).transpose(1, 2)
    vc = rand((B, Lk, Hkv, 128), 3).transpose(1, 2)
    out, lse = ops.decode_attention(q.to(dev), kc.to(dev), vc.to(dev))
    o_ref, l_ref = orc.cpu_sdpa_forward(q, kc, vc)
    orc.assert_close_bf16(out, o_ref, "out")
    orc.assert_close_lse(lse, l_ref)
    qq = rand((B, 4, 1, 128), 4)
    kk = rand((B, 4, 300, 128), 5)
    res = ops._scaled_dot_product_flash_attention(qq.to(dev), kk.to(dev), kk.to(dev))
    o_ref, l_ref = orc.cpu_sdpa_forward(qq, kk, kk)
    orc.assert_close_bf16(res[0], o_ref, "out")
    orc.assert_close_lse(res[1][..., :1], l_ref)  # the operator pads the logsumexp to 16 rows


def test_decode_split_count_does_not_change_the_answer_much(cuda_device, native_lib):
    """Size-independent property at the benchmark's KV length: any split count gives the same
    result up to fp32 merge rounding, and equals the oracle on a sampled batch element."""
    dev = cuda_device
    c = workloads.config5_decode(batch=4, seqlen_k=32768)
    q, k, v = c.q.to(dev), c.k.to(dev), c.v.to(dev)
    base_o, base_l = ops.decode_attention(q, k, v, scale=c.softmax_scale, num_splits=1)
    for s in (0, 7, 16, 64):
        o, l = ops.decode_attention(q, k, v, scale=c.softmax_scale, num_splits=s)
        assert orc.error_stats(o, base_o)[0] <= 2e-3
        assert orc.error_stats(l, base_l)[0] <= 2e-6
    o_ref, l_ref = orc.cpu_sdpa_forward(c.q[1:2], c.k[1:2], c.v[1:2], scale=c.softmax_scale)
    orc.assert_close_bf16(base_o[1:2], o_ref, "out")
    orc.assert_close_lse(base_l[1:2], l_ref)


@pytest.mark.parametrize("head_stride", [3, 12345])
def test_decode_with_one_head_takes_any_head_stride(cuda_device, native_lib, head_stride):
    dev = cuda_device
    q, buf = rand((2, 4, 1, 128), 1).to(dev), rand((2, 70, 128), 2).to(dev)
    k = buf[:, :64].unsqueeze(1)
    odd = k.as_strided(k.shape, (k.stride(0), head_stride, k.stride(2), 1))
    out, lse = ops.decode_attention(q, odd, odd)
    want, want_lse = ops.decode_attention(q, k, k)
    assert torch.equal(out, want) and torch.equal(lse, want_lse)


@pytest.mark.parametrize("B,Hq,Hkv,Lk,D", [(4, 32, 8, 32768, 128), (16, 32, 8, 8192, 128), (8, 16, 4, 20000, 64), (1, 32, 8, 1000, 128)])
def test_decode_error_against_64_bits(cuda_device, native_lib, B, Hq, Hkv, Lk, D):
    """The weights and the result are rounded to bf16, whose rounding to nearest has a relative error of 1.53e-3 (2-norm, mantissas
    spread evenly over the logarithm): 2.17e-3 for both, less what the weights of exactly 1 save. However long the share of a CTA
    is, the largest weight of every 16 keys is one of those."""
    g = torch.Generator(device=cuda_device).manual_seed(5)
    q, k, v = (torch.randn(B, h, n, D, generator=g, device=cuda_device).bfloat16() for h, n in ((Hq, 1), (Hkv, Lk), (Hkv, Lk)))
    out, lse = ops.decode_attention(q, k, v)
    assert ops.device_status() == 0
    err = ref_norm = 0.0
    for b in range(B):
        s = torch.einsum("hgd,hkd->hgk", q[b].double().view(Hkv, Hq // Hkv, D), k[b].double()) * D ** -0.5
        want = torch.einsum("hgk,hkd->hgd", s.softmax(-1), v[b].double()).reshape(Hq, 1, D)
        err += float((out[b].double() - want).norm() ** 2)
        ref_norm += float(want.norm() ** 2)
    assert (err / ref_norm) ** 0.5 <= 2.05e-3, (err / ref_norm) ** 0.5
