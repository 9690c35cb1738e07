"""The work that users of this package have it do, as cases that can be timed and compared.

A case is a dict of plain values; its ``kind`` says which public call it stands for:

  prefill   causal attention over whole prompts (``LocalStrideSparseAttention``)
  padded    the same over a left-padded batch (``left_paddings``)
  varlen    packed prompts under a user-defined per-head block pattern (``SparseAttention``)
  chunked   a serving step: prompt chunks and decode tokens packed in one call
  decode    one query token per sequence against a left-padded K/V cache
  train     forward and backward, gradients for q, k and v

``listed()`` are the cases themselves, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program holds before the call, ``run`` is the call.
"""
import math
import random

import numpy as np
import torch

from dkernel_b200 import LocalStrideSparseAttention, SparseAttention

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# The local + vertical-stride pattern of the package's benchmark: 64-token blocks, a band of 16 blocks,
# one block column in 8.
PHI3 = {"block": 64, "local": 16, "stride": 8}


def listed():
    return [
        # Batched prefill at the benchmark's shape: what a prompt-processing server does all day.
        dict(name="prefill", kind="prefill", dtype="bf16", batch=4, seq=8192, hq=32, hkv=8, dim=128, max_seq=8192,
             lse=True, **PHI3),
        # One short prompt of an odd length (an interactive request): latency counts.
        dict(name="prefill_short", kind="prefill", dtype="bf16", batch=1, seq=517, hq=32, hkv=8, dim=128,
             max_seq=8192, lse=False, **PHI3),
        # One long document.
        dict(name="prefill_long", kind="prefill", dtype="fp16", batch=1, seq=32768, hq=32, hkv=8, dim=128,
             max_seq=32768, lse=False, **PHI3),
        # Small heads and 32-token blocks: the finer patterns of the test matrix.
        dict(name="prefill_block32", kind="prefill", dtype="fp16", batch=2, seq=4000, hq=16, hkv=16, dim=64,
             max_seq=4096, lse=True, block=32, local=16, stride=8),
        # Prompts of different lengths, left-padded to the longest, as batched generation starts.
        dict(name="padded", kind="padded", dtype="bf16", batch=8, seq=2048, lo=256, lens=1, hq=32, hkv=8, dim=128,
             max_seq=8192, lse=False, **PHI3),
        # Packed prompts under a random pattern of its own for every head.
        dict(name="varlen", kind="varlen", dtype="bf16", batch=16, lo=512, hi=4096, lens=2, hq=32, hkv=32, dim=128,
             max_seq=16384, density=0.2, block=64),
        # One step of a continuous-batching server: prompt chunks beside decode tokens.
        dict(name="chunked", kind="chunked", dtype="bf16", chunks=3, chunk=512, tokens=45, hi=8192, lens=3, hq=32,
             hkv=8, dim=128, max_seq=16384, **PHI3),
        # Batched decode at the benchmark's shape, and the same step on an 8-bit cache.
        dict(name="decode", kind="decode", dtype="bf16", fp8=False, batch=64, seq=8192, lo=1024, lens=4, hq=32, hkv=8,
             dim=128, max_seq=8192, **PHI3),
        dict(name="decode_fp8", kind="decode", dtype="bf16", fp8=True, batch=64, seq=8192, lo=1024, lens=5, hq=32,
             hkv=8, dim=128, max_seq=8192, **PHI3),
        # One user's token: the smallest call there is.
        dict(name="decode_one", kind="decode", dtype="bf16", fp8=False, batch=1, seq=4096, lo=3000, lens=6, hq=32,
             hkv=8, dim=128, max_seq=8192, **PHI3),
        # Training step at the benchmark's shape.
        dict(name="train", kind="train", dtype="bf16", batch=2, seq=8192, hq=32, hkv=32, dim=128, max_seq=8192,
             block=64, local=32, stride=8),
        # Training of a small model: grouped heads, narrow head dim, an odd sequence length.
        dict(name="train_small", kind="train", dtype="fp16", batch=4, seq=1500, hq=16, hkv=4, dim=64, max_seq=2048,
             block=64, local=8, stride=4),
    ]


# (q heads, kv heads, head dim)
HEADS = [(32, 8, 128), (32, 8, 128), (32, 32, 128), (16, 4, 64), (16, 16, 64), (24, 8, 96)]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
    kind = rng.choice(["prefill", "prefill", "padded", "varlen", "chunked", "decode", "decode", "decode", "train", "train"])
    hq, hkv, dim = rng.choice(HEADS)
    c = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "fp16"]), hq=hq, hkv=hkv, dim=dim,
             block=rng.choice([64, 64, 64, 32, 128]), local=rng.choice([4, 8, 16, 32]), stride=rng.choice([4, 8, 16]))
    if kind in ("prefill", "train"):
        c.update(batch=_log(rng, 1, 8), seq=_log(rng, 64, 32768 if kind == "prefill" else 8192))
        c["max_seq"] = -(-c["seq"] // 2048) * 2048
        if kind == "prefill":
            c["lse"] = rng.random() < 0.5
    elif kind == "padded":
        c.update(batch=_log(rng, 2, 16), seq=_log(rng, 128, 8192), lens=rng.randrange(1 << 20), lse=rng.random() < 0.5)
        c["lo"] = max(1, c["seq"] // rng.choice([2, 8]))
        c["max_seq"] = -(-c["seq"] // 2048) * 2048
    elif kind == "varlen":
        hi = _log(rng, 256, 8192)
        c.update(block=64, batch=_log(rng, 1, 32), lo=hi // 8, hi=hi, lens=rng.randrange(1 << 20),
                 max_seq=-(-hi // 4096) * 4096, density=rng.choice([0.1, 0.2, 0.4]), hkv=rng.choice([hq, hkv]))
        del c["local"], c["stride"]
    elif kind == "chunked":
        c.update(block=64, chunks=rng.randint(1, 6), chunk=64 * _log(rng, 2, 32), tokens=_log(rng, 1, 96),
                 hi=_log(rng, 1024, 16384), lens=rng.randrange(1 << 20), max_seq=32768)
    else:
        # the decode kernel's head dims and blocks; a cache of `seq` slots, `lo` the shortest context
        c.update(hq=32, hkv=rng.choice([8, 8, 4, 32]), dim=rng.choice([128, 128, 64]), block=rng.choice([64, 64, 128]),
                 fp8=rng.random() < 0.4, batch=_log(rng, 1, 96), seq=_log(rng, 512, 32768), lens=rng.randrange(1 << 20))
        c["lo"] = max(1, c["seq"] // rng.choice([2, 8]))
        c["max_seq"] = -(-c["seq"] // 8192) * 8192
    return c


def draw(rng):
    """One more case; drawn again while it would cost more than the largest listed ones."""
    flops = max(work(c)["flops"] for c in listed())
    cache = 64 * 8192 * 8 * 128            # slots x kv heads x dim of the benchmark's decode cache
    while True:
        c = _draw(rng)
        slots = {"decode": lambda: c["batch"] * c["seq"], "chunked": lambda: sum(k for _, k in _lengths(c))}
        if c["kind"] in slots and slots[c["kind"]]() * c["hkv"] * c["dim"] > cache:
            continue
        w = work(c)
        if w["flops"] <= (flops if c["kind"] == "train" else flops / 2) and w["bytes"] <= 1e9:
            return c


# ------------------------------------------------------------------ lengths and patterns of a case
def _lengths(c):
    """[(q_len, k_len)] of the case's sequences; the same for every seed, so that work() knows them."""
    kind = c["kind"]
    if kind in ("prefill", "train"):
        return [(c["seq"], c["seq"])] * c["batch"]
    r = random.Random(c["lens"])
    if kind == "padded":
        lens = [r.randint(c["lo"], c["seq"]) for _ in range(c["batch"] - 1)] + [c["seq"]]
        return [(n, n) for n in lens]
    if kind == "varlen":
        return [(n, n) for n in (r.randint(c["lo"], c["hi"]) for _ in range(c["batch"]))]
    if kind == "decode":
        return [(1, r.randint(c["lo"], c["seq"])) for _ in range(c["batch"])]
    # chunked: chunks start on block boundaries of their prompt; decode tokens anywhere
    out = []
    for _ in range(c["chunks"]):
        past = r.randrange(0, max(1, c["hi"] // c["block"])) * c["block"]
        n = c["chunk"] if r.random() < 0.7 else r.randint(1, c["chunk"])      # the last chunk of a prompt is ragged
        out.append((n, past + n))
    out += [(1, r.randint(16, c["hi"])) for _ in range(c["tokens"])]
    return out


def _user_pattern(c):
    """uint8 (hq, blocks, blocks): a random lower triangle with the diagonal set, another for every head."""
    n = c["max_seq"] // c["block"]
    p = np.random.RandomState(c["lens"]).random_sample((c["hq"], n, n)) < c["density"]
    return (np.tril(p) | np.eye(n, dtype=bool)[None]).astype(np.uint8)


def _row_counts(c):
    """(q heads that each counted head stands for, [head][row] attended blocks left of the diagonal)."""
    if c["kind"] == "varlen":
        return 1, _user_pattern(c).sum(-1, dtype=np.int64) - 1
    n = -(-c["max_seq"] // c["block"])
    row, col = np.arange(n)[:, None], np.arange(n)[None, :]
    heads = []
    step = max(1, c["stride"] // c["hq"])
    for kvh in range(min(c["hkv"], c["stride"])):
        on = ((row - col < c["local"]) | ((col + kvh * step) % c["stride"] == 0)) & (col < row)
        heads.append(on.sum(-1))
    return c["hq"] / len(heads), np.array(heads, dtype=np.int64)


def work(c):
    bs = c["block"]
    times, counts = _row_counts(c)
    pairs = q_tok = k_tok = 0
    for q_len, k_len in _lengths(c):
        pos = np.arange(k_len - q_len, k_len)
        keys = counts[:, pos // bs] * bs + (pos % bs + 1)       # attended keys of every query token
        pairs += float(keys.sum()) * times
        q_tok += q_len
        # a single query token needs only the keys it attends, counted per kv head
        k_tok += k_len if q_len > 1 else float(keys.sum()) * times / c["hq"]
    d = c["dim"]
    q_bytes = q_tok * c["hq"] * d * 2
    kv_bytes = k_tok * c["hkv"] * d * 2 * (1 if c.get("fp8") else 2)
    if c["kind"] == "train":
        # q, k, v, dO in; o, dq, dk, dv out; two products forward and five backward
        return {"bytes": 4 * q_bytes + 2 * kv_bytes, "flops": 14.0 * d * pairs}
    lse = q_tok * c["hq"] * 4 if c.get("lse") else 0
    return {"bytes": 2 * q_bytes + kv_bytes + lse, "flops": 4.0 * d * pairs}


def tolerance(c):
    # Against the same inputs widened to 32 bits, with 32-bit sums (the package's CUDA-core kernels), the
    # calls show (2-norm, largest): bf16 outputs 2.1e-3 and 0.035, gradients 2.5e-3 and 0.17; fp16 outputs
    # 2.9e-4 and 0.0036, gradients 3.2e-4 and 0.010.  Stated is four times that.
    bf16 = c["dtype"] == "bf16"
    if c["kind"] == "train":
        return {"rel": 1e-2, "max": 0.68} if bf16 else {"rel": 1.3e-3, "max": 0.04}
    return {"rel": 8.4e-3, "max": 0.14} if bf16 else {"rel": 1.2e-3, "max": 0.015}


# ------------------------------------------------------------------ inputs and the call
def _module(c):
    if c["kind"] == "varlen":
        return SparseAttention(c["block"], torch.from_numpy(_user_pattern(c)).cuda())
    return LocalStrideSparseAttention(c["hq"], c["max_seq"], c["block"], c["local"], c["stride"], num_kv_heads=c["hkv"],
                                      seq_dim=1)


def prepare(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dt = DTYPES[c["dtype"]]

    def randn(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dt)

    hq, hkv, d = c["hq"], c["hkv"], c["dim"]
    s = {"kind": c["kind"], "attn": _module(c), "scale": 1.0 / math.sqrt(d), "lse": bool(c.get("lse"))}
    lens = _lengths(c)
    if c["kind"] in ("varlen", "chunked"):
        q_lens, k_lens = zip(*lens)
        s["cu_q"] = torch.tensor(np.cumsum((0,) + q_lens), dtype=torch.int32, device="cuda")
        s["cu_k"] = torch.tensor(np.cumsum((0,) + k_lens), dtype=torch.int32, device="cuda")
        s["q"], s["k"], s["v"] = randn(sum(q_lens), hq, d), randn(sum(k_lens), hkv, d), randn(sum(k_lens), hkv, d)
        return s
    b, n = c["batch"], c["seq"]
    s["q"] = randn(b, 1 if c["kind"] == "decode" else n, hq, d)
    s["k"], s["v"] = randn(b, n, hkv, d), randn(b, n, hkv, d)
    if c["kind"] in ("padded", "decode"):
        s["left"] = torch.tensor([n - k for _, k in lens], dtype=torch.int32, device="cuda")
    if c.get("fp8"):
        # stored with one scale per tensor, the largest value near the top of the format's range
        s["scales"] = (8.0 / 448.0, 8.0 / 448.0)
        s["k"] = (s["k"].float() / s["scales"][0]).to(torch.float8_e4m3fn)
        s["v"] = (s["v"].float() / s["scales"][1]).to(torch.float8_e4m3fn)
    if c["kind"] == "train":
        s["do"] = randn(b, n, hq, d)
        for x in ("q", "k", "v"):
            s[x].requires_grad_()
    return s


def run(s):
    kind = s["kind"]
    attn, q, k, v, scale = s["attn"], s["q"], s["k"], s["v"], s["scale"]
    if kind == "train":
        out = attn(q, k, v, sm_scale=scale)
        return (out.detach(), *torch.autograd.grad(out, (q, k, v), s["do"]))
    with torch.no_grad():
        if kind == "prefill":
            return attn(q, k, v, sm_scale=scale, return_lse=s["lse"])
        if kind == "padded":
            return attn(q, k, v, sm_scale=scale, left_paddings=s["left"], return_lse=s["lse"])
        if kind == "decode":
            if "scales" in s:
                return attn(q, k, v, sm_scale=scale, left_paddings=s["left"], kv_scales=s["scales"])
            return attn(q, k, v, sm_scale=scale, left_paddings=s["left"])
        if kind == "varlen":
            return attn(q, k, v, sm_scale=scale, cu_seqlen_k=s["cu_k"])
        return attn(q, k, v, sm_scale=scale, cu_seqlen_k=s["cu_k"], cu_seqlen_q=s["cu_q"])
