"""Performance cases of the attention library: what its users have it do, with sizes over the whole range of use.

A case is a dict of plain values. ``kind`` says which public call it makes:

* ``decode``   one new token per sequence against a K/V cache: ``ops.decode_attention``
* ``prefill``  dense forward, also with a cached prefix (more keys than queries): ``ops.gqa_prefill``
* ``varlen``   packed sequences, forward: ``ops._flash_attention_forward``
* ``train``    dense forward + backward: ``F.scaled_dot_product_attention`` with the aten operators pointed at this
  library (``via`` "torch"), or the package's own ``sdp_choice.scaled_dot_product_attention`` (``via`` "package");
  ``extra`` adds dropout, a boolean key-padding mask or a learned relative-position bias
* ``varlen_train``  packed sequences, forward + backward: the registered operator ``b200_sdpa::_flash_attention_forward``

Inputs are N(0,1) in the case's 16-bit type, as activations behind a normalisation are. ``layout`` "blhd" makes q, k, v the
transposed views of [batch, sequence, heads, head_dim] tensors that a model's projections produce, "bhld" contiguous ones.
"""
import math
import random

import torch
import torch.nn.functional as F

from torch_mlu_b200 import backends, ops, sdp_choice, torch_glue

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    return [
        # one interactive sequence, early in its answer: a few microseconds of work, all latency
        dict(name="decode_b1_l1000", kind="decode", batch=1, heads_q=32, heads_kv=8, len_k=1000, head_dim=128, dtype="bf16"),
        # a full serving batch at 32 K tokens of context: 8 GiB of K and V per pass (the benchmark's decode workload)
        dict(name="decode_b64_l32768", kind="decode", batch=64, heads_q=32, heads_kv=8, len_k=32768, head_dim=128, dtype="bf16"),
        # the smallest configuration: an encoder layer on short sentences
        dict(name="prefill_b2_h8_l256_d64", kind="prefill", batch=2, heads_q=8, heads_kv=8, len_q=256, len_k=256, head_dim=64,
             causal=False, dtype="bf16", layout="bhld"),
        # the headline workload: causal prefill of a 32-head model
        dict(name="prefill_b4_h32_l4096", kind="prefill", batch=4, heads_q=32, heads_kv=32, len_q=4096, len_k=4096, head_dim=128,
             causal=True, dtype="bf16", layout="bhld"),
        # chunked prefill: the next 512 tokens of two prompts whose first 7680 tokens are in the cache
        dict(name="prefill_chunk512_of_8192", kind="prefill", batch=2, heads_q=32, heads_kv=8, len_q=512, len_k=8192,
             head_dim=128, causal=True, dtype="bf16", layout="bhld"),
        # a serving batch of sixteen packed prompts of 512 to 4096 tokens, GQA (the benchmark's packed workload)
        dict(name="varlen_16seq_512_4096", kind="varlen", seqs=16, lo=512, hi=4096, lens_seed=3, heads_q=32, heads_kv=8,
             head_dim=128, causal=True, dtype="bf16"),
        # a small model's training step on sequences of an odd length, through torch's own entry point
        dict(name="train_b4_h8_l500_d64_f16", kind="train", via="torch", extra="none", batch=4, heads=8, length=500, head_dim=64,
             causal=False, dtype="f16", layout="blhd"),
        # the benchmark's training workload
        dict(name="train_b8_h16_l2048", kind="train", via="package", extra="none", batch=8, heads=16, length=2048, head_dim=128,
             causal=True, dtype="bf16", layout="bhld"),
        # the same with dropout
        dict(name="train_b8_h16_l2048_drop", kind="train", via="package", extra="dropout", batch=8, heads=16, length=2048,
             head_dim=128, causal=True, dtype="bf16", layout="bhld"),
        # encoder training with a key-padding mask
        dict(name="train_b8_h12_l512_d64_mask", kind="train", via="package", extra="mask", batch=8, heads=12, length=512,
             head_dim=64, causal=False, dtype="bf16", layout="blhd"),
        # fine-tuning on packed sequences of very different lengths, GQA
        dict(name="varlen_train_12seq_64_2048", kind="varlen_train", seqs=12, lo=64, hi=2048, lens_seed=7, heads_q=16, heads_kv=4,
             head_dim=128, causal=True, dtype="bf16"),
        # head_dim 256 training (the benchmark's workload)
        dict(name="train_b4_h16_l4096_d256", kind="train", via="package", extra="none", batch=4, heads=16, length=4096,
             head_dim=256, causal=True, dtype="bf16", layout="bhld"),
    ]


# The largest cost of a drawn case of each kind, in bytes and operations: those of the largest listed one.
MOST_BYTES = {"decode": 8.7e9, "prefill": 1e9, "varlen": 1e9, "train": 2e9, "varlen_train": 1e9}
MOST_FLOPS = {"decode": 1e12, "prefill": 5.6e11, "varlen": 8.1e11, "train": 1.95e12, "varlen_train": 5e11}


def _log_int(rng, lo, hi):
    """An integer between lo and hi, evenly spread over the logarithm: mostly odd ones, some multiples of 64."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.4:
        n = max(64, n // 64 * 64)
    return max(lo, min(hi, n))


def draw(rng):
    while True:
        kind = rng.choice(["decode", "prefill", "prefill", "varlen", "train", "train", "train", "varlen_train"])
        dtype = rng.choice(["bf16", "bf16", "f16"])
        heads_q, heads_kv = rng.choice([(32, 8), (32, 8), (16, 16), (32, 32), (16, 4), (64, 8), (8, 1), (12, 12)])
        if kind == "decode":
            case = dict(kind=kind, batch=_log_int(rng, 1, 64), heads_q=heads_q, heads_kv=heads_kv, len_k=_log_int(rng, 64, 32768),
                        head_dim=rng.choice([128, 128, 64]), dtype=dtype)
        elif kind == "prefill":
            len_q = _log_int(rng, 64, 8192)
            prefix = _log_int(rng, 64, 8192) if rng.random() < 0.3 else 0
            case = dict(kind=kind, batch=_log_int(rng, 1, 8), heads_q=heads_q, heads_kv=heads_kv, len_q=len_q,
                        len_k=len_q + prefix, head_dim=rng.choice([128, 128, 64, 96, 256]), causal=prefix > 0 or rng.random() < 0.7,
                        dtype=dtype, layout=rng.choice(["bhld", "blhd"]))
        elif kind in ("varlen", "varlen_train"):
            lo = _log_int(rng, 16, 1024)
            case = dict(kind=kind, seqs=_log_int(rng, 2, 32), lo=lo, hi=_log_int(rng, 2 * lo, 4096), lens_seed=rng.randrange(10000),
                        heads_q=heads_q, heads_kv=heads_kv, head_dim=rng.choice([128, 128, 64]), causal=rng.random() < 0.8,
                        dtype=dtype)
        else:
            extra = rng.choice(["none", "none", "none", "dropout", "mask", "bias"])
            length = _log_int(rng, 64, 8192 if extra == "none" else 2048)
            head_dim = rng.choice([128, 128, 64, 64, 80] + ([256, 192] if extra in ("none", "dropout") else []))
            case = dict(kind=kind, via=rng.choice(["torch", "package"]) if extra == "none" and head_dim <= 128 else "package",
                        extra=extra, batch=_log_int(rng, 1, 16), heads=rng.choice([8, 12, 16, 32]), length=length,
                        head_dim=head_dim, causal=extra in ("none", "dropout") and rng.random() < 0.7, dtype=dtype,
                        layout=rng.choice(["bhld", "blhd"]))
        w = work(case)
        if w["bytes"] <= MOST_BYTES[kind] and w["flops"] <= MOST_FLOPS[kind]:
            return case


def _lengths(case):
    r = random.Random(case["lens_seed"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["seqs"])]


def _randn(gen, dtype, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)


def _heads_first(gen, case, heads, length):
    """A [batch, heads, length, head_dim] tensor in the case's memory layout."""
    b, d, dt = case["batch"], case["head_dim"], DTYPES[case["dtype"]]
    if case["layout"] == "blhd":
        return _randn(gen, dt, b, length, heads, d).transpose(1, 2)
    return _randn(gen, dt, b, heads, length, d)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dt, d = case["kind"], DTYPES[case["dtype"]], case["head_dim"]
    s = dict(case)
    if kind == "decode":
        s["q"] = _randn(gen, dt, case["batch"], case["heads_q"], 1, d)
        for name in ("k", "v"):
            s[name] = _randn(gen, dt, case["batch"], case["heads_kv"], case["len_k"], d)
    elif kind == "prefill":
        s["q"] = _heads_first(gen, case, case["heads_q"], case["len_q"])
        for name in ("k", "v"):
            s[name] = _heads_first(gen, case, case["heads_kv"], case["len_k"])
    elif kind in ("varlen", "varlen_train"):
        lens = _lengths(case)
        ends = [sum(lens[:i]) for i in range(len(lens) + 1)]
        s["cu"] = torch.tensor(ends, dtype=torch.int32, device="cuda")
        s["longest"] = max(lens)
        for name, heads in (("q", case["heads_q"]), ("k", case["heads_kv"]), ("v", case["heads_kv"])):
            s[name] = _randn(gen, dt, ends[-1], heads, d)
        if kind == "varlen_train":
            torch_glue.load()
            s["dout"] = _randn(gen, dt, ends[-1], case["heads_q"], d)
            for name in ("q", "k", "v"):
                s[name].requires_grad_()
    else:
        for name in ("q", "k", "v"):
            s[name] = _heads_first(gen, case, case["heads"], case["length"]).requires_grad_()
        s["dout"] = _randn(gen, dt, case["batch"], case["length"], case["heads"], d).transpose(1, 2)
        s["mask"] = None
        if case["via"] == "torch":
            # once, at a program's start: torch's operators run this library, and its flash backend is the one that is used
            torch_glue.install_aten_overrides()
            backends.enable_flash_sdp(True)
            backends.enable_mem_efficient_sdp(False)
            backends.enable_math_sdp(False)
            torch.backends.cuda.enable_cudnn_sdp(False)
        else:
            backends.enable_flash_sdp(True)
            backends.enable_mem_efficient_sdp(True)
            backends.enable_math_sdp(False)
            torch_glue.load()
        if case["extra"] == "dropout":
            torch.cuda.manual_seed(seed)  # the pattern is drawn from the device's default generator
        elif case["extra"] == "mask":
            n = torch.randint(case["length"] // 2, case["length"] + 1, (case["batch"], 1, 1, 1), generator=gen, device="cuda")
            s["mask"] = torch.arange(case["length"], device="cuda").view(1, 1, 1, -1) < n
        elif case["extra"] == "bias":
            s["mask"] = _randn(gen, dt, 1, case["heads"], case["length"], case["length"]).requires_grad_()
    return s


def run(s):
    kind = s["kind"]
    if kind == "decode":
        return ops.decode_attention(s["q"], s["k"], s["v"])
    if kind == "prefill":
        return ops.gqa_prefill(s["q"], s["k"], s["v"], is_causal=s["causal"])
    if kind == "varlen":
        return ops._flash_attention_forward(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"], 0.0, s["causal"],
                                            False)[:2]
    if kind == "varlen_train":
        out = torch.ops.b200_sdpa._flash_attention_forward(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["longest"], s["longest"],
                                                           0.0, s["causal"], False)[0]
        return out.detach(), *torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["dout"])
    sdpa = F.scaled_dot_product_attention if s["via"] == "torch" else sdp_choice.scaled_dot_product_attention
    out = sdpa(s["q"], s["k"], s["v"], attn_mask=s["mask"], dropout_p=0.1 if s["extra"] == "dropout" else 0.0,
               is_causal=s["causal"])
    wanted = (s["q"], s["k"], s["v"]) + ((s["mask"],) if s["extra"] == "bias" else ())
    return out.detach(), *torch.autograd.grad(out, wanted, s["dout"])


def _visible_pairs(len_q, len_k, causal):
    """(query, key) pairs that the mask leaves, bottom-right aligned as in a cached prefix."""
    return len_q * (len_k - len_q) + len_q * (len_q + 1) // 2 if causal else len_q * len_k


def work(case):
    """Forward: two products over the visible pairs, q, k, v in and out and logsumexp out. Backward: five products (scores once
    more), q, k, v, out, dout and logsumexp in and three gradients out. A padding mask hides keys of a share that the seed
    decides: every key counts here."""
    kind, d = case["kind"], case["head_dim"]
    if kind == "decode":
        rows_q, rows_k = case["batch"] * case["heads_q"], case["batch"] * case["heads_kv"] * case["len_k"]
        pairs = rows_q * case["len_k"]
    elif kind == "prefill":
        rows_q = case["batch"] * case["heads_q"] * case["len_q"]
        rows_k = case["batch"] * case["heads_kv"] * case["len_k"]
        pairs = case["batch"] * case["heads_q"] * _visible_pairs(case["len_q"], case["len_k"], case["causal"])
    elif kind in ("varlen", "varlen_train"):
        lens = _lengths(case)
        rows_q, rows_k = case["heads_q"] * sum(lens), case["heads_kv"] * sum(lens)
        pairs = case["heads_q"] * sum(_visible_pairs(n, n, case["causal"]) for n in lens)
    else:
        rows_q = rows_k = case["batch"] * case["heads"] * case["length"]
        pairs = case["batch"] * case["heads"] * _visible_pairs(case["length"], case["length"], case["causal"])
    total = (2 * rows_q + 2 * rows_k) * d * 2 + rows_q * 4
    flops = 4 * pairs * d
    if kind in ("train", "varlen_train"):
        total += (4 * rows_q + 4 * rows_k) * d * 2 + rows_q * 4
        flops += 10 * pairs * d
        if case.get("extra") == "bias":  # read by the forward and the backward, its gradient written
            total += 3 * case["heads"] * case["length"] ** 2 * 2
    return {"bytes": total, "flops": flops}


def tolerance(case):
    # the probabilities and the results are rounded to the 16-bit type, sums are fp32
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
