"""Padded, packed (varlen) and decode routes vs the CPU oracle."""
import math

import numpy as np
import pytest
import torch

from oracle import dkernel_oracle as O
from helpers import assert_out_close, assert_lse_close, seeded_qkv

pytestmark = pytest.mark.gpu


def _module(Hq, max_seq, pk, **kw):
    from dkernel_b200 import LocalStrideSparseAttention
    pk = dict(pk)
    return LocalStrideSparseAttention.__wrapped__(Hq, max_seq, pk.pop("block_size"), pk.pop("local_blocks"),
                                                  pk.pop("vert_stride"), **pk, **kw)


@pytest.mark.parametrize("B,Hq,Hkv,S,D,dtype,seq_dim,pk,right", [
    (3, 4, 2, 320, 64, torch.float16, 1, dict(block_size=64, local_blocks=2, vert_stride=3, num_kv_heads=2), False),
    (2, 2, 2, 512, 128, torch.bfloat16, 2, dict(block_size=64, local_blocks=2, vert_stride=4, homo_head=True), False),
    (3, 2, 2, 300, 128, torch.bfloat16, 1, dict(block_size=64, local_blocks=3, vert_stride=2), True),
    (2, 2, 2, 256, 32, torch.float32, 1, dict(block_size=16, local_blocks=4, vert_stride=4), False),
])
def test_padded_prefill(B, Hq, Hkv, S, D, dtype, seq_dim, pk, right):
    bs = pk["block_size"]
    shape = (lambda h: (B, h, S, D)) if seq_dim == 2 else (lambda h: (B, S, h, D))
    q, k, v = seeded_qkv(11, shape(Hq), shape(Hkv), dtype)
    lens = torch.randint(1, S, (B,), generator=torch.Generator().manual_seed(2))
    lens[0] = S
    bm = O.block_mask(Hq, S, **pk)
    mod = _module(Hq, S, pk, seq_dim=seq_dim)
    if right:
        ref, ref_lse = O.padded_attention(q.float(), k.float(), v.float(), bm, bs, seqlens=lens, seq_dim=seq_dim)
        out, lse = mod(q.cuda(), k.cuda(), v.cuda(), seqlens=lens.cuda(), return_lse=True)
    else:
        left = S - lens
        ref, ref_lse = O.padded_attention(q.float(), k.float(), v.float(), bm, bs, left_paddings=left,
                                          seq_dim=seq_dim)
        out, lse = mod(q.cuda(), k.cuda(), v.cuda(), left_paddings=left.cuda(), return_lse=True)
    tight = dtype == torch.float32
    assert_out_close(out, ref, max_abs=2e-4 if tight else 2e-2, mean_abs=2e-5 if tight else 2e-3)
    assert_lse_close(lse, ref_lse, tol=1e-4 if tight else 1e-3)


@pytest.mark.parametrize("Hq,Hkv,D,dtype,bs,lens", [
    (4, 4, 128, torch.bfloat16, 64, [512, 100, 333, 64, 1]),
    (4, 2, 64, torch.float16, 32, [200, 31, 256]),
    (2, 2, 128, torch.bfloat16, 64, [700]),
])
def test_varlen_prefill_user_pattern(Hq, Hkv, D, dtype, bs, lens):
    """Packed sequences with a random lower-triangular user pattern (config-5 style)."""
    from dkernel_b200 import SparseAttention
    nb = 16
    g = torch.Generator().manual_seed(0)
    pat = torch.rand(Hq, nb, nb, generator=g) < 0.3
    pat |= torch.eye(nb, dtype=torch.bool)[None]
    pat &= torch.tril(torch.ones(nb, nb, dtype=torch.bool))[None]
    T = sum(lens)
    q, k, v = seeded_qkv(5, (T, Hq, D), (T, Hkv, D), dtype)
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32)
    ref, ref_lse = O.varlen_attention(q.float(), k.float(), v.float(), cu, pat.numpy().astype(np.uint8), bs)
    with pytest.warns(UserWarning):
        mod = SparseAttention(bs, pat.cuda())
    out, lse = mod(q.cuda(), k.cuda(), v.cuda(), cu_seqlen_k=cu.cuda(), return_lse=True)
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)


@pytest.mark.parametrize("impl", ["sm100", "generic"])
def test_varlen_batched_chunked_prefill(impl):
    """A packed batch that mixes whole prompts, decode tokens and prompt chunks whose earlier
    part is already in the KV cache (q_len not in {1, k_len}; the chunk starts on a block
    boundary).  The reference's kernel computes this case (pattern row from past_len + q
    offset, dkernel/ops/sparse_attn_inference.py:507-514) but its host code refuses it
    (:211-212); here the host does not look at the lengths, so it is served."""
    from dkernel_b200 import SparseAttention
    Hq, Hkv, D, bs, nb = 8, 2, 128, 64, 16
    g = torch.Generator().manual_seed(3)
    pat = torch.rand(Hq, nb, nb, generator=g) < 0.35
    pat |= torch.eye(nb, dtype=torch.bool)[None]
    pat &= torch.tril(torch.ones(nb, nb, dtype=torch.bool))[None]
    q_lens = [64, 1, 130, 72, 300]
    k_lens = [192, 300, 130, 200, 940]          # pasts 128, 299, 0, 128, 640
    cu_q = torch.tensor([0] + list(np.cumsum(q_lens)), dtype=torch.int32)
    cu_k = torch.tensor([0] + list(np.cumsum(k_lens)), dtype=torch.int32)
    q, k, v = seeded_qkv(31, (sum(q_lens), Hq, D), (sum(k_lens), Hkv, D), torch.bfloat16)
    ref, ref_lse = O.varlen_attention(q.float(), k.float(), v.float(), cu_k, pat.numpy().astype(np.uint8), bs,
                                      cu_seqlens_q=cu_q)
    with pytest.warns(UserWarning):
        mod = SparseAttention(bs, pat.cuda(), impl=impl)
    out, lse = mod(q.cuda(), k.cuda(), v.cuda(), cu_seqlen_k=cu_k.cuda(), cu_seqlen_q=cu_q.cuda(),
                   return_lse=True)
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)


@pytest.mark.parametrize("B,Hq,Hkv,S,D,dtype,seq_dim,pk,bps", [
    (5, 8, 2, 1024, 128, torch.bfloat16, 1, dict(block_size=64, local_blocks=4, vert_stride=4, num_kv_heads=2), 0),
    (3, 4, 4, 640, 64, torch.float16, 2, dict(block_size=64, local_blocks=2, vert_stride=3), 2),
    (2, 4, 1, 1024, 128, torch.bfloat16, 1, dict(block_size=128, local_blocks=2, vert_stride=2, num_kv_heads=1), 1),
    (2, 2, 2, 256, 32, torch.float32, 1, dict(block_size=32, local_blocks=2, vert_stride=2), 0),   # generic route
])
def test_left_padded_decode(B, Hq, Hkv, S, D, dtype, seq_dim, pk, bps):
    bs = pk["block_size"]
    kshape = (B, Hkv, S, D) if seq_dim == 2 else (B, S, Hkv, D)
    qshape = (B, Hq, 1, D) if seq_dim == 2 else (B, 1, Hq, D)
    q, k, v = seeded_qkv(13, qshape, kshape, dtype)
    lens = torch.randint(1, S + 1, (B,), generator=torch.Generator().manual_seed(4))
    lens[0] = S
    lens[-1] = 1
    left = S - lens
    bm = O.block_mask(Hq, S, **pk)
    q1 = q if seq_dim == 1 else q.transpose(1, 2)
    k1, v1 = (k, v) if seq_dim == 1 else (k.transpose(1, 2), v.transpose(1, 2))
    ref, ref_lse = O.decode_attention(q1.float(), k1.float(), v1.float(), bm, bs, left_paddings=left)
    if seq_dim == 2:
        ref = ref.transpose(1, 2)
    mod = _module(Hq, S, pk, seq_dim=seq_dim)
    if bps:
        from dkernel_b200.ops import decode
        out, lse = decode(q.cuda(), k.cuda(), v.cuda(), mod._plan(), 1 / math.sqrt(D), seq_dim=seq_dim,
                          k_start=left.to(torch.int32).cuda(),
                          k_end=torch.full((B,), S, dtype=torch.int32).cuda(), blocks_per_split=bps)
        lse = lse.unsqueeze(-1)
    else:
        out, lse = mod(q.cuda(), k.cuda(), v.cuda(), left_paddings=left.cuda(), return_lse=True)
    tight = dtype == torch.float32
    assert_out_close(out, ref, max_abs=2e-4 if tight else 2e-2, mean_abs=2e-5 if tight else 2e-3)
    assert_lse_close(lse, ref_lse, tol=1e-4 if tight else 1e-3)


def test_unpadded_and_packed_decode():
    B, Hq, Hkv, S, D, bs = 2, 4, 2, 64 * 5 + 12, 128, 64
    pk = dict(block_size=bs, local_blocks=2, vert_stride=3, num_kv_heads=Hkv)
    q, k, v = seeded_qkv(17, (B, 1, Hq, D), (B, S, Hkv, D), torch.bfloat16)
    bm = O.block_mask(Hq, 1024, **pk)
    ref, ref_lse = O.decode_attention(q.float(), k.float(), v.float(), bm, bs)
    mod = _module(Hq, 1024, pk, seq_dim=1)
    out, lse = mod(q.cuda(), k.cuda(), v.cuda(), return_lse=True)
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)
    # packed: q (B, Hq, D), k/v (sum lens, Hkv, D)
    lens = [S, 77]
    kp = torch.cat([k[0, :lens[0]], k[1, :lens[1]]])
    vp = torch.cat([v[0, :lens[0]], v[1, :lens[1]]])
    cu = torch.tensor([0, lens[0], lens[0] + lens[1]], dtype=torch.int32)
    refp, _ = O.varlen_attention(q[:, 0].float(), kp.float(), vp.float(), cu, bm, bs)
    outp = mod(q[:, 0].cuda(), kp.cuda(), vp.cuda(), cu_seqlen_k=cu.cuda())
    assert_out_close(outp, refp)


def test_kv_sharded_decode_merges_to_whole():
    """KV shards by position range + combine_attn_partitions == un-sharded decode."""
    from dkernel_b200.ops import decode
    from dkernel_b200 import combine_attn_partitions
    B, Hq, Hkv, S, D, bs = 4, 8, 2, 1024, 128, 64
    pk = dict(block_size=bs, local_blocks=4, vert_stride=4, num_kv_heads=Hkv)
    q, k, v = seeded_qkv(19, (B, 1, Hq, D), (B, S, Hkv, D), torch.bfloat16)
    lens = torch.tensor([1024, 700, 65, 300])
    left = S - lens
    bm = O.block_mask(Hq, S, **pk)
    ref, ref_lse = O.decode_attention(q.float(), k.float(), v.float(), bm, bs, left_paddings=left)
    mod = _module(Hq, S, pk, seq_dim=1)
    G = 2
    parts = []
    for r in range(G):
        # rank r holds, for every sequence, positions [lo, hi) (block aligned), left-packed locally
        nblk = (lens + bs - 1) // bs
        lo = (nblk * r // G) * bs
        hi = torch.minimum((nblk * (r + 1) // G) * bs, lens)
        n = (hi - lo).clamp_min(0)
        cap = int(n.max().item())
        ks = torch.zeros(B, max(cap, 1), Hkv, D, dtype=k.dtype)
        vs = torch.zeros_like(ks)
        for b in range(B):
            s0 = int(left[b] + lo[b])
            ks[b, :int(n[b])] = k[b, s0:s0 + int(n[b])]
            vs[b, :int(n[b])] = v[b, s0:s0 + int(n[b])]
        o, l = decode(q.cuda(), ks.cuda(), vs.cuda(), mod._plan(), 1 / math.sqrt(D), seq_dim=1,
                      k_start=torch.zeros(B, dtype=torch.int32).cuda(), k_end=n.to(torch.int32).cuda(),
                      k_pos0=lo.to(torch.int32).cuda(), k_total=lens.to(torch.int32).cuda())
        parts.append((o, l.unsqueeze(-1)))
    merged, mlse = combine_attn_partitions(*parts, hdim=2, return_lse=True)
    assert_out_close(merged, ref)
    assert_lse_close(mlse, ref_lse)


@pytest.mark.parametrize("W", [2, 4, 8])
def test_block_cyclic_kv_shards_merge_to_whole(W):
    """Block-cyclic KV shards (block j of a sequence on rank j % W) decoded one rank after the
    other on this GPU + combine_attn_partitions == un-sharded decode; ranks without any attended
    block give O = 0, LSE = -inf."""
    from dkernel_b200.ops import decode
    from dkernel_b200.dist import kv_shard_cyclic_blocks, pack_kv_shard_cyclic
    from dkernel_b200 import combine_attn_partitions
    B, Hq, Hkv, S, D, bs = 5, 8, 2, 2048, 128, 64
    pk = dict(block_size=bs, local_blocks=6, vert_stride=4, num_kv_heads=Hkv)
    q, k, v = seeded_qkv(29, (B, 1, Hq, D), (B, S, Hkv, D), torch.bfloat16)
    lens = torch.tensor([2048, 700, 65, 1, 1300])
    left = S - lens
    bm = O.block_mask(Hq, S, **pk)
    ref, ref_lse = O.decode_attention(q.float(), k.float(), v.float(), bm, bs, left_paddings=left)
    mod = _module(Hq, S, pk, seq_dim=1)
    parts, stored = [], torch.zeros_like(lens)
    for r in range(W):
        ks, vs, n = pack_kv_shard_cyclic(k, v, left, lens, r, W, bs)
        assert torch.equal(n, kv_shard_cyclic_blocks(lens, r, W, bs))
        stored += n
        o, l = decode(q.cuda(), ks.cuda(), vs.cuda(), mod._plan(), 1 / math.sqrt(D), seq_dim=1,
                      k_end=n.to(torch.int32).cuda(), k_total=lens.to(torch.int32).cuda(), k_blk=(W, r))
        parts.append((o, l.unsqueeze(-1)))
    assert torch.equal(stored, lens)                       # every token lives on exactly one rank
    merged, mlse = combine_attn_partitions(*parts, hdim=2, return_lse=True)
    assert_out_close(merged, ref)
    assert_lse_close(mlse, ref_lse)
    from dkernel_b200 import _lib
    assert _lib.wait_status() == 0


@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (64, torch.bfloat16), (128, torch.float16)])
def test_decode_reads_an_e4m3_kv_cache(D, dtype):
    """K/V stored as float8_e4m3fn with per-tensor scales: the decode kernel converts the stored
    bytes exactly, so the result must equal the oracle on the de-quantised cache -- left padding,
    right padding, the split-KV path (long rows) and a packed batch."""
    from dkernel_b200 import SparseAttention
    B, Hq, Hkv, S, bs = 5, 8, 2, 2048, 64
    pk = dict(block_size=bs, local_blocks=6, vert_stride=4, num_kv_heads=Hkv)
    q, k, v = seeded_qkv(61, (B, 1, Hq, D), (B, S, Hkv, D), dtype)
    ks, vs = float(k.float().abs().max()) / 448.0, float(v.float().abs().max()) / 448.0
    k8 = (k.float() / ks).to(torch.float8_e4m3fn)
    v8 = (v.float() / vs).to(torch.float8_e4m3fn)
    kd, vd = k8.float() * ks, v8.float() * vs                  # what the cache stands for
    bm = O.block_mask(Hq, S, **pk)
    mod = _module(Hq, S, pk, seq_dim=1)
    lens = torch.tensor([2048, 700, 65, 1, 1300])
    left = S - lens
    ref, ref_lse = O.decode_attention(q.float(), kd, vd, bm, bs, left_paddings=left)
    with torch.no_grad():
        out, lse = mod(q.cuda(), k8.cuda(), v8.cuda(), left_paddings=left.cuda(), return_lse=True,
                       kv_scales=(ks, vs))
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)
    # right padding: whatever follows the sequence in the cache is ignored (0xff bytes are NaN in e4m3)
    k8r, v8r = k8.clone(), v8.clone()
    for b in range(B):
        k8r[b, int(lens[b]):].view(torch.uint8).fill_(0xff)
        v8r[b, int(lens[b]):].view(torch.uint8).fill_(0xff)
    ref, ref_lse = O.decode_attention(q.float(), kd, vd, bm, bs, seqlens=lens)
    with torch.no_grad():
        out, lse = mod(q.cuda(), k8r.cuda(), v8r.cuda(), seqlens=lens.cuda(), return_lse=True, kv_scales=(ks, vs))
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)
    # packed batch, one query token per sequence
    lens2 = [300, 64, 1, 999]
    cu = torch.tensor([0] + list(np.cumsum(lens2)), dtype=torch.int32)
    T = int(cu[-1])
    kp, vp = seeded_qkv(62, (T, Hkv, D), (T, Hkv, D), dtype)[:2]
    kp8, vp8 = (kp.float() / ks).to(torch.float8_e4m3fn), (vp.float() / vs).to(torch.float8_e4m3fn)
    qp = q[:4, 0]
    refp, _ = O.varlen_attention(qp.float(), kp8.float() * ks, vp8.float() * vs, cu, bm, bs)
    with torch.no_grad():
        outp = mod(qp.cuda(), kp8.cuda(), vp8.cuda(), cu_seqlen_k=cu.cuda(), kv_scales=(ks, vs))
    assert_out_close(outp, refp)
    # an 8-bit cache without scales, or on a prefill call, is refused before any launch
    with pytest.raises(AssertionError):
        mod(q.cuda(), k8.cuda(), v8.cuda(), left_paddings=left.cuda())
    with pytest.raises(AssertionError):
        mod(q.expand(B, 1, Hq, D).repeat(1, S, 1, 1).cuda(), k8.cuda(), v8.cuda(), kv_scales=(ks, vs))
    from dkernel_b200 import _lib
    assert _lib.wait_status() == 0


def test_sharded_decode_single_rank_group(tmp_path):
    """sharded_decode end to end (packed (O, LSE) rows -> all-gather -> fused merge) with a
    one-rank NCCL group: the whole sequence is the only shard."""
    import torch.distributed as dist
    from dkernel_b200.dist import sharded_decode
    B, Hq, Hkv, S, D, bs = 3, 8, 2, 1024, 128, 64
    pk = dict(block_size=bs, local_blocks=4, vert_stride=4, num_kv_heads=Hkv)
    q, k, v = seeded_qkv(23, (B, 1, Hq, D), (B, S, Hkv, D), torch.bfloat16)
    lens = torch.tensor([1024, 513, 64])
    bm = O.block_mask(Hq, S, **pk)
    # left-aligned storage: sequence b occupies rows [0, lens[b])
    ref, ref_lse = O.decode_attention(q.float(), k.float(), v.float(), bm, bs, seqlens=lens)
    mod = _module(Hq, S, pk, seq_dim=1)
    store = dist.FileStore(str(tmp_path / "pg"), 1)
    dist.init_process_group("nccl", store=store, rank=0, world_size=1)
    try:
        out, lse = sharded_decode(mod, q.cuda(), k.cuda(), v.cuda(), lens.to(torch.int32).cuda(),
                                  torch.zeros(B, dtype=torch.int32).cuda(), lens.to(torch.int32).cuda(),
                                  1 / math.sqrt(D))
        torch.cuda.synchronize()
    finally:
        dist.destroy_process_group()
    assert_out_close(out, ref)
    assert_lse_close(lse.unsqueeze(-1), ref_lse)


def test_combine_attn_partitions_matches_reference_fixture(golden_dir):
    from dkernel_b200 import combine_attn_partitions
    C = np.load(f"{golden_dir}/combine.npz")
    parts = [(torch.from_numpy(C[f"o{i}"]).cuda(), torch.from_numpy(C[f"lse{i}"]).cuda()) for i in range(3)]
    res = combine_attn_partitions(*parts)
    assert (res.cpu() - torch.from_numpy(C["combined"])).abs().max().item() < 1e-5
    # hdim = 2 (outputs laid out (B, S, H, D))
    parts2 = [(o.transpose(1, 2).contiguous(), l) for o, l in parts]
    res2 = combine_attn_partitions(*parts2, hdim=2)
    assert (res2.transpose(1, 2).cpu() - torch.from_numpy(C["combined"])).abs().max().item() < 1e-5
    # -inf partitions contribute nothing and do not create NaN
    o0, l0 = parts[0]
    dead = (torch.full_like(o0, float("nan")).nan_to_num(0.0), torch.full_like(l0, float("-inf")))
    res3, lse3 = combine_attn_partitions(parts[0], dead, return_lse=True)
    assert (res3 - o0).abs().max().item() < 1e-6 and (lse3 - l0).abs().max().item() < 1e-6
    # differentiable route gives the same numbers and gradients reach the LSEs
    pg = [(o.clone().requires_grad_(), l.clone().requires_grad_()) for o, l in parts]
    r = combine_attn_partitions(*pg)
    assert (r.detach().cpu() - torch.from_numpy(C["combined"])).abs().max().item() < 1e-5
    r.sum().backward()
    assert pg[0][1].grad is not None and torch.isfinite(pg[0][1].grad).all()


def test_seq_partition_equivalence():
    """Chunked q x kv attention merged by LSE equals the un-partitioned result
    (the reference's tests/test_seq_partition.py, 'ring' and 'one-kv' modes), forward
    and backward."""
    from dkernel_b200 import SparseAttention, get_sparse_attn_mask, combine_attn_partitions
    b, h, S, d, bs, nparts = 1, 3, 1024, 64, 64, 4
    dtype = torch.bfloat16
    for mode in ("ring", "one-kv"):
        q, k, v, do = seeded_qkv(20, (b, h, S, d), (b, h, S, d), dtype, device="cuda", with_do=True)
        q.requires_grad_(), k.requires_grad_(), v.requires_grad_()
        chunk = S // nparts
        outs = []
        for qc in range(nparts):
            end_kv = (qc + 1) * chunk
            ranges = [(i * chunk, (i + 1) * chunk) for i in range(qc + 1)] if mode == "ring" else [(0, end_kv)]
            parts, masks = [], []
            for (ks, ke) in ranges:
                _, bmask, _ = get_sparse_attn_mask(h, chunk, bs, 4, 4, dtype=torch.uint8,
                                                   q_start_position=qc * chunk, kv_start_position=ks,
                                                   kv_seqlen=ke - ks)
                masks.append(bmask)
                layer = SparseAttention(bs, bmask, seq_dim=2, causal=(ke == end_kv))
                parts.append(layer(q[:, :, qc * chunk:end_kv], k[:, :, ks:ke], v[:, :, ks:ke], return_lse=True))
            outs.append(parts[0][0] if len(parts) == 1 else combine_attn_partitions(*parts, hdim=1))
            _, full, _ = get_sparse_attn_mask(h, S, bs, 4, 4, dtype=torch.uint8)
            cat = torch.cat(masks, dim=-1)
            assert (cat == full[:, qc * (chunk // bs):(qc + 1) * (chunk // bs), :cat.size(-1)]).all()
        out = torch.cat(outs, dim=2)
        out.backward(do)
        grads = [t.grad.clone() for t in (q, k, v)]
        for t in (q, k, v):
            t.grad = None
        _, full, _ = get_sparse_attn_mask(h, S, bs, 4, 4, dtype=torch.uint8)
        ref_layer = SparseAttention(bs, full, seq_dim=2)
        ref = ref_layer(q, k, v)
        ref.backward(do)
        assert torch.allclose(out, ref, rtol=1e-2, atol=1e-2), mode
        for g, t, n in zip(grads, (q, k, v), "qkv"):
            assert torch.allclose(g, t.grad, rtol=1e-2, atol=2e-2), f"{mode} d{n}: {(g - t.grad).abs().max()}"
            t.grad = None


@pytest.mark.parametrize("n_seq,k_len", [(17, 4096), (65, 1025)])
def test_packed_batch_with_more_than_64k_keys_runs_on_tensor_cores(n_seq, k_len):
    """The 65536-key limit of the tensor-core forward is one sequence's, not the packed batch's: chunks and
    decode tokens of contexts that together hold more keys stay on it (no fall-back warning) and are right."""
    import warnings
    Hq, Hkv, D, bs = 4, 2, 64, 64
    q_lens = [1 if i % 3 else 33 for i in range(n_seq)]
    k_lens = [k_len if n % 2 else (k_len // bs) * bs + n for n in q_lens]      # chunks start on a block boundary
    k_lens = [(kl // bs) * bs + ql if ql > 1 else kl for kl, ql in zip(k_lens, q_lens)]
    assert sum(k_lens) > 65536
    pk = dict(block_size=bs, local_blocks=3, vert_stride=5, num_kv_heads=Hkv)
    cu_q = torch.tensor([0] + list(np.cumsum(q_lens)), dtype=torch.int32)
    cu_k = torch.tensor([0] + list(np.cumsum(k_lens)), dtype=torch.int32)
    q, k, v = seeded_qkv(41, (sum(q_lens), Hq, D), (sum(k_lens), Hkv, D), torch.bfloat16)
    bm = O.block_mask(Hq, 8192, **pk)
    ref, ref_lse = O.varlen_attention(q.float(), k.float(), v.float(), cu_k, bm, bs, cu_seqlens_q=cu_q)
    mod = _module(Hq, 8192, pk, impl="sm100")
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        out, lse = mod(q.cuda(), k.cuda(), v.cuda(), cu_seqlen_k=cu_k.cuda(), cu_seqlen_q=cu_q.cuda(), return_lse=True)
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("Hq,Hkv,D,bs,dtype,q_gain", [
    (4, 4, 128, 64, torch.bfloat16, 1.0),     # one head per group
    (6, 2, 64, 64, torch.float16, 8.0),       # logits that move the reference maximum
    (8, 1, 128, 128, torch.bfloat16, 8.0),    # a full 8-column tile
    (12, 1, 128, 64, torch.float16, 1.0),     # two column tiles, the second one half empty
    (32, 2, 64, 128, torch.bfloat16, 1.0),    # two full column tiles
])
def test_decode_group_sizes_and_unit_edges(fp8, Hq, Hkv, D, bs, dtype, q_gain):
    """Lengths around the edges of the decode kernel's 32- and 64-token units and of the pattern's blocks,
    for every number of heads per group that changes how its products are tiled.  The oracle gets the
    stored (rounded) K/V, so the bounds are those of the 16-bit products: the helpers' defaults."""
    lens = [1, 31, 32, 33, 63, 64, 65, 127, 129, 257, 500]
    B, S = len(lens), 512
    pk = dict(block_size=bs, local_blocks=2, vert_stride=3, num_kv_heads=Hkv)
    q, k, v = seeded_qkv(61, (B, 1, Hq, D), (B, S, Hkv, D), dtype)
    q = q * q_gain
    scales, kw = (0.02, 0.015), {}
    if fp8:
        k, v = (k.float() / scales[0]).to(torch.float8_e4m3fn), (v.float() / scales[1]).to(torch.float8_e4m3fn)
        kw["kv_scales"] = scales
    kf, vf = (k.float() * scales[0], v.float() * scales[1]) if fp8 else (k.float(), v.float())
    left = torch.tensor([S - n for n in lens], dtype=torch.int32)
    ref, ref_lse = O.decode_attention(q.float(), kf, vf, O.block_mask(Hq, S, **pk), bs, left_paddings=left)
    mod = _module(Hq, S, pk, seq_dim=1)
    with torch.no_grad():
        out, lse = mod(q.cuda(), k.cuda(), v.cuda(), left_paddings=left.cuda(), return_lse=True, **kw)
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)


@pytest.mark.parametrize("Hq,Hkv,S,D,bs,seq_dim,lens,right", [
    (4, 2, 300, 128, 64, 1, [300, 1, 64, 65, 130], False),      # two heads per tile
    (2, 2, 320, 40, 64, 2, [1, 127, 128, 129, 319], True),      # two row blocks per tile, five pieces a row
    (4, 4, 257, 64, 32, 1, [63, 256, 191, 2], False),           # fine blocks
    (2, 1, 130, 256, 64, 2, [5, 130], True),
])
def test_pad_rows_of_a_padded_batch_are_written(Hq, Hkv, S, D, bs, seq_dim, lens, right):
    """The output comes from uninitialised memory: every pad row must be written (zeros, LSE -inf), whatever
    the memory held; an output that the caller brings keeps its pad rows."""
    pk = dict(block_size=bs, local_blocks=2, vert_stride=3)
    B = len(lens)
    shape = (lambda h: (B, h, S, D)) if seq_dim == 2 else (lambda h: (B, S, h, D))
    q, k, v = seeded_qkv(71, shape(Hq), shape(Hkv), torch.bfloat16)
    n = torch.tensor(lens)
    kw = dict(seqlens=n) if right else dict(left_paddings=S - n)
    ref, ref_lse = O.padded_attention(q.float(), k.float(), v.float(), O.block_mask(Hq, S, num_kv_heads=Hkv, **pk), bs,
                                      seq_dim=seq_dim, **kw)
    mod = _module(Hq, S, dict(pk, num_kv_heads=Hkv), seq_dim=seq_dim, impl="sm100")
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    kw = {a: t.cuda() for a, t in kw.items()}
    for _ in range(2):
        dirty = [torch.full_like(q, float("nan")), torch.full((B, Hq, S), float("nan"), device="cuda")]
        del dirty      # back to the caching allocator, which hands the blocks out again
        with torch.no_grad():
            out, lse = mod(q, k, v, return_lse=True, **kw)
        assert_out_close(out, ref)
        assert_lse_close(lse, ref_lse)
        assert ((ref == 0).all(-1) == (out.cpu() == 0).all(-1)).all()
    own = torch.full_like(q, 7.0)
    mod_out = _module(Hq, S, dict(pk, num_kv_heads=Hkv), seq_dim=seq_dim, impl="sm100", out=own)
    with torch.no_grad():
        mod_out(q, k, v, **kw)
    pad = (ref == 0).all(-1)
    assert (own.cpu()[pad] == 7.0).all() and torch.equal(own.cpu()[~pad], out.cpu()[~pad])


@pytest.mark.parametrize("Hq,Hkv,D,dtype,user_pattern", [
    (8, 2, 128, torch.bfloat16, False),     # four heads of a group in one decode CTA
    (4, 4, 64, torch.float16, False),
    (4, 2, 128, torch.bfloat16, True),      # a pattern per q head: one head per decode CTA
    (24, 2, 64, torch.bfloat16, False),     # twelve heads: two column tiles
    (4, 2, 96, torch.float16, False),       # not a head dim of the decode kernel
])
def test_packed_single_token_sequences_beside_chunks(Hq, Hkv, D, dtype, user_pattern):
    """One packed call with empty sequences, single query tokens and chunks, more than 32 sequences: single
    tokens run on the decode kernel, the rest on the prefill kernel, and every row of the output is written."""
    from dkernel_b200 import SparseAttention
    bs, S = 64, 4096
    g = torch.Generator().manual_seed(4)
    if user_pattern:
        nb = S // bs
        pat = torch.tril(torch.rand(Hq, nb, nb, generator=g) < 0.3) | torch.eye(nb, dtype=torch.bool)[None]
        bm, mod = pat.numpy(), SparseAttention(bs, pat.to(torch.uint8).cuda(), impl="sm100")
    else:
        pk = dict(block_size=bs, local_blocks=3, vert_stride=4, num_kv_heads=Hkv)
        bm, mod = O.block_mask(Hq, S, **pk), _module(Hq, S, pk, impl="sm100")
    q_lens = [1, 130, 0, 1, 64, 1] + [1] * 30 + [63, 1]
    k_lens = [1, 130, 0, 64, 128, 65] + [1 + int(x) for x in torch.randint(0, 900, (30,), generator=g)] + [191, 4096]
    cu_q = torch.tensor(np.cumsum([0] + q_lens), dtype=torch.int32)
    cu_k = torch.tensor(np.cumsum([0] + k_lens), dtype=torch.int32)
    q, k, v = seeded_qkv(81, (sum(q_lens), Hq, D), (sum(k_lens), Hkv, D), dtype)
    ref, ref_lse = O.varlen_attention(q.float(), k.float(), v.float(), cu_k, bm, bs, cu_seqlens_q=cu_q)
    dirty = torch.full_like(q, float("nan")).cuda()
    del dirty
    with torch.no_grad():
        out, lse = mod(q.cuda(), k.cuda(), v.cuda(), cu_seqlen_k=cu_k.cuda(), cu_seqlen_q=cu_q.cuda(), return_lse=True)
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("Hq,Hkv,D,bps", [(4, 1, 128, 9), (4, 1, 128, 4), (8, 8, 64, 3), (16, 1, 128, 2), (4, 2, 128, 1)])
def test_decode_split_counts(fp8, Hq, Hkv, D, bps):
    """Two to eight splits of a row are merged inside a cluster, more (the last case) by a second launch; rows
    with fewer blocks than splits leave some CTAs without work."""
    from dkernel_b200.ops import decode
    bs, lens = 64, [1, 64, 65, 200, 640, 1024, 1000]
    B, S = len(lens), 1024
    pk = dict(block_size=bs, local_blocks=16, vert_stride=4, num_kv_heads=Hkv)      # dense: up to 16 blocks a row
    q, k, v = seeded_qkv(91, (B, 1, Hq, D), (B, S, Hkv, D), torch.bfloat16)
    scales = (0.02, 0.015) if fp8 else None
    if fp8:
        k, v = (k.float() / scales[0]).to(torch.float8_e4m3fn), (v.float() / scales[1]).to(torch.float8_e4m3fn)
    kf, vf = (k.float() * scales[0], v.float() * scales[1]) if fp8 else (k.float(), v.float())
    left = torch.tensor([S - n for n in lens], dtype=torch.int32)
    ref, ref_lse = O.decode_attention(q.float(), kf, vf, O.block_mask(Hq, S, **pk), bs, left_paddings=left)
    mod = _module(Hq, S, pk, seq_dim=1)
    out, lse = decode(q.cuda(), k.cuda(), v.cuda(), mod._plan(), 1.0 / math.sqrt(D), seq_dim=1, k_start=left.cuda(),
                      blocks_per_split=bps, kv_scales=scales)
    assert_out_close(out, ref)
    assert_lse_close(lse.unsqueeze(-1), ref_lse)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("scale", [-0.09, 0.0])
@pytest.mark.parametrize("Hq,Hkv,D,dtype,bps", [
    (4, 1, 128, torch.bfloat16, 0),     # splits merged inside a cluster
    (4, 2, 64, torch.float16, 16),      # one split
    (12, 1, 64, torch.bfloat16, 1),     # two column tiles, splits merged by a second launch
])
def test_decode_with_a_scale_that_is_not_positive(fp8, scale, Hq, Hkv, D, dtype, bps):
    """The sign of the scale turns the order of the logits round, and scale 0 makes all of them equal: in full
    units (the reference maximum) and in partial ones (the mask), on padded and packed caches.  Logits spread
    over +-40, so that a reference taken from the wrong end overflows.  Bounds: the helpers' defaults."""
    from dkernel_b200.ops import decode
    bs, S, lens = 64, 1024, [1, 31, 33, 63, 64, 65, 200, 1000, 1024]
    B = len(lens)
    pk = dict(block_size=bs, local_blocks=16, vert_stride=4, num_kv_heads=Hkv)      # dense: up to 16 blocks a row
    q, k, v = seeded_qkv(93, (B, 1, Hq, D), (B, S, Hkv, D), dtype)
    q = q * 8
    scales, kw = (0.02, 0.015), {}
    if fp8:
        k, v = (k.float() / scales[0]).to(torch.float8_e4m3fn), (v.float() / scales[1]).to(torch.float8_e4m3fn)
        kw["kv_scales"] = scales
    kf, vf = (k.float() * scales[0], v.float() * scales[1]) if fp8 else (k.float(), v.float())
    left = torch.tensor([S - n for n in lens], dtype=torch.int32)
    ref, ref_lse = O.decode_attention(q.float(), kf, vf, O.block_mask(Hq, S, **pk), bs, sm_scale=scale, left_paddings=left)
    mod = _module(Hq, S, pk, seq_dim=1)
    out, lse = decode(q.cuda(), k.cuda(), v.cuda(), mod._plan(), scale, seq_dim=1, k_start=left.cuda(),
                      blocks_per_split=bps, **kw)
    assert_out_close(out, ref)
    assert_lse_close(lse.unsqueeze(-1), ref_lse)
    cu = torch.tensor(np.cumsum([0] + lens), dtype=torch.int32).cuda()
    kp, vp = (torch.cat([t[i, S - n:].view(torch.uint8) for i, n in enumerate(lens)]).view(t.dtype) for t in (k, v))
    out, lse = decode(q[:, 0].cuda(), kp.cuda(), vp.cuda(), mod._plan(), scale, seq_dim=None, k_start=cu[:-1], k_end=cu[1:],
                      blocks_per_split=bps, **kw)
    assert_out_close(out, ref[:, 0])
    assert_lse_close(lse.unsqueeze(-1), ref_lse)


@pytest.mark.parametrize("n", [40, 64])
def test_negative_scale_decode_is_the_last_row_of_the_prefill(n):
    """One module, one scale: the token that a decode step computes is the last one of the prefill."""
    pk = dict(block_size=64, local_blocks=2, vert_stride=3, num_kv_heads=2)
    q, k, v = (t.cuda() for t in seeded_qkv(95, (1, n, 4, 64), (1, n, 2, 64), torch.float16))
    mod = _module(4, 512, pk, seq_dim=1)
    left = torch.zeros(1, dtype=torch.int32, device="cuda")
    with torch.no_grad():
        pre = mod(q, k, v, sm_scale=-0.2, left_paddings=left)
        out = mod(q[:, -1:].contiguous(), k, v, sm_scale=-0.2, left_paddings=left)
    assert_out_close(out, pre[:, -1:])


@pytest.mark.parametrize("Hq,Hkv,D,extra", [(4, 2, 128, 0), (2, 2, 72, 4), (4, 2, 256, 0), (2, 1, 16, 12)])
def test_pad_rows_of_empty_sequences_and_of_unaligned_outputs(Hq, Hkv, D, extra):
    """A sequence of nothing but pads, and pad rows of an output whose rows start 8 bytes off a 16-byte boundary
    (``extra`` elements behind every row, which must keep what they hold).  The kernel's own real rows are the
    reference's (an aligned output), the pad rows zero, LSE -inf."""
    from dkernel_b200 import _lib, ops
    B, S, bs = 4, 200, 64
    pk = dict(block_size=bs, local_blocks=2, vert_stride=3, num_kv_heads=Hkv)
    q, k, v = (t.cuda() for t in seeded_qkv(97, (B, S, Hq, D), (B, S, Hkv, D), torch.bfloat16))
    left = torch.tensor([S, 0, S - 1, 77], dtype=torch.int32, device="cuda")
    plan = _module(Hq, 256, pk, seq_dim=1)._plan()
    buf = torch.full((B, S, Hq, D + extra), 7.0, dtype=q.dtype, device="cuda")
    o, lse = buf[..., :D], torch.full((B, Hq, S), float("nan"), device="cuda")
    ends = torch.full((B,), S, dtype=torch.int32, device="cuda")
    p = ops._fwd_params(q, k, v, o, lse, 1, plan, 0.1, True, _lib.ROWS_BY_POSITION_ZERO_PADS, left, ends, left, ends,
                        impl=_lib.IMPL_SM100)
    ops._launch_fwd(p, q)
    ref, ref_lse = O.padded_attention(q.float().cpu(), k.float().cpu(), v.float().cpu(), O.block_mask(Hq, 256, **pk), bs,
                                      sm_scale=0.1, left_paddings=left.cpu())
    assert_out_close(o, ref)
    assert_lse_close(lse, ref_lse)
    pad = torch.arange(S, device="cuda")[None] < left[:, None]
    assert (o[pad] == 0).all() and torch.isneginf(lse.transpose(1, 2)[pad]).all()
    assert (buf[..., D:] == 7.0).all()


def _launches(fn):
    """Number of nodes of the graph that a call of fn is captured into."""
    import ctypes
    fn()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    n = ctypes.c_size_t(0)
    assert ctypes.CDLL("libcuda.so.1").cuGraphGetNodes(ctypes.c_void_p(g.raw_cuda_graph()), None, ctypes.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("q_lens,k_lens,second", [
    ([64], [192], False),                                  # one chunk
    ([65, 1, 1], [193, 700, 33], False),                   # too few sequences
    ([1, 64, 130, 1], [1, 64, 130, 1], False),             # whole prompts (as many queries as keys)
    ([65, 1, 0, 1], [193, 700, 0, 33], True),
    ([64, 64, 64, 64, 64], [64, 128, 192, 256, 320], True),   # chunks only: the launch finds nothing to do
    ([1, 1, 1, 1, 1], [1, 64, 65, 128, 511], True),           # no tile at all
])
def test_packed_call_launches_the_single_token_kernel_where_it_pays(q_lens, k_lens, second):
    """A packed batch whose query ranges cannot hold single decode tokens, or few of them, is one launch; both routes
    give the oracle's rows, and what follows in the stream sees them."""
    Hq, Hkv, D, bs, S = 8, 2, 64, 64, 1024
    pk = dict(block_size=bs, local_blocks=3, vert_stride=4, num_kv_heads=Hkv)
    mod = _module(Hq, S, pk, impl="sm100")
    cu_q = torch.tensor(np.cumsum([0] + q_lens), dtype=torch.int32)
    cu_k = torch.tensor(np.cumsum([0] + k_lens), dtype=torch.int32)
    q, k, v = seeded_qkv(99, (sum(q_lens), Hq, D), (sum(k_lens), Hkv, D), torch.bfloat16)
    ref, ref_lse = O.varlen_attention(q.float(), k.float(), v.float(), cu_k, O.block_mask(Hq, S, **pk), bs, cu_seqlens_q=cu_q)
    q, k, v, cu_q, cu_k = (t.cuda() for t in (q, k, v, cu_q, cu_k))

    def call(return_lse=False):
        with torch.no_grad():
            return mod(q, k, v, cu_seqlen_k=cu_k, cu_seqlen_q=cu_q, return_lse=return_lse)
    out, lse = call(True)
    assert_out_close(out.clone(), ref)
    assert_lse_close(lse, ref_lse)
    assert _launches(call) == (2 if second else 1)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("Hq,Hkv,D,dtype", [
    (3, 1, 128, torch.bfloat16), (8, 2, 64, torch.bfloat16), (4, 4, 128, torch.float16),      # lo terms in idle columns
    (6, 1, 64, torch.float16), (8, 1, 128, torch.bfloat16),                                    # ... as a second product
    (12, 1, 128, torch.bfloat16), (9, 1, 64, torch.float16), (16, 1, 64, torch.float16),        # two column tiles
])
def test_decode_weights_keep_their_fp32_value(fp8, Hq, Hkv, D, dtype):
    """fp32 partials (no rounding of the output) against 64 bits.  Two 16-bit terms leave 2^-18 of a weight, the
    fp32 logits (up to 2^4) and exponentials a few 2^-20; one term alone would show 2^-9 / sqrt(3) = 1.1e-3 (bf16)
    or 1.4e-4 (f16)."""
    from dkernel_b200.ops import decode
    bs, lens = 64, [1, 63, 64, 200, 777, 1024]
    B, S = len(lens), 1024
    pk = dict(block_size=bs, local_blocks=16, vert_stride=4, num_kv_heads=Hkv)      # dense rows of 16 blocks
    q, k, v = (t.cuda() for t in seeded_qkv(101, (B, 1, Hq, D), (B, S, Hkv, D), dtype))
    scales, kw = (1.0, 1.0), {}
    if fp8:
        scales = (0.02, 0.015)
        k, v, kw = (k.float() / scales[0]).to(torch.float8_e4m3fn), (v.float() / scales[1]).to(torch.float8_e4m3fn), dict(kv_scales=scales)
    left = torch.tensor([S - n for n in lens], dtype=torch.int32, device="cuda")
    o, _ = decode(q, k, v, _module(Hq, S, pk, seq_dim=1)._plan(), 1.0 / math.sqrt(D), seq_dim=1, k_start=left,
                  blocks_per_split=16, partials_only=True, **kw)
    k, v = (t.double().repeat_interleave(Hq // Hkv, 2) * s for t, s in zip((k, v), scales))
    ref = torch.empty(B, Hq, D, dtype=torch.float64, device="cuda")
    for i, n in enumerate(lens):
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i, 0].double(), k[i, S - n:]) / math.sqrt(D), -1)
        ref[i] = torch.einsum("hn,nhd->hd", p, v[i, S - n:])
    err = (o.view(B, Hq, D).double() - ref).norm() / ref.norm()
    assert err <= 2e-5, float(err)


@pytest.mark.parametrize("D,bs,dtype", [(64, 64, torch.bfloat16), (128, 64, torch.float16), (256, 64, torch.bfloat16),
                                        (128, 32, torch.bfloat16), (64, 16, torch.float16)])
def test_packed_batch_with_more_than_64k_keys_keeps_fp32_weights(D, bs, dtype):
    """Such calls were computed in fp32 before the tensor cores took them.  Against 64 bits their error is the rounding
    of the output and nothing else worth the name (5 %); 16-bit weights would add 40 % to it."""
    Hq, Hkv, S, n_seq = 2, 1, 4096, 17
    pk = dict(block_size=bs, local_blocks=256 // bs, vert_stride=5, num_kv_heads=Hkv)
    mod = _module(Hq, S, pk, impl="sm100")
    q_lens = [1 if i % 3 == 0 else 67 if i % 3 == 1 else 64 for i in range(n_seq)]
    k_lens = [(3840 if n > 1 else 4000) + n for n in q_lens]          # chunks start on a block boundary
    assert sum(k_lens) > 65536
    q, k, v = (t.cuda() for t in seeded_qkv(103, (sum(q_lens), Hq, D), (sum(k_lens), Hkv, D), dtype))
    cu_q, cu_k = (torch.tensor(np.cumsum([0] + n), dtype=torch.int32, device="cuda") for n in (q_lens, k_lens))
    with torch.no_grad():
        out = mod(q, k, v, cu_seqlen_k=cu_k, cu_seqlen_q=cu_q)
    bm = torch.from_numpy(np.asarray(O.block_mask(Hq, S, **pk)).astype(bool)).cuda()
    ref = torch.empty(out.shape, dtype=torch.float64, device="cuda")
    for i, (nq, nk) in enumerate(zip(q_lens, k_lens)):
        rows, keys = slice(int(cu_q[i]), int(cu_q[i + 1])), slice(int(cu_k[i]), int(cu_k[i + 1]))
        qpos, kpos = torch.arange(nk - nq, nk, device="cuda"), torch.arange(nk, device="cuda")
        for h in range(Hq):
            on = bm[h % bm.size(0)][(qpos // bs)[:, None], (kpos // bs)[None]] & (kpos[None] <= qpos[:, None])
            a = q[rows, h].double() @ k[keys, 0].double().T / math.sqrt(D)
            ref[rows, h] = torch.softmax(a.masked_fill(~on, -math.inf), -1) @ v[keys, 0].double()
    err, rounding = (out.double() - ref).norm(), (ref.to(dtype).double() - ref).norm()
    assert err <= 1.05 * rounding, float(err / rounding)


@pytest.mark.parametrize("many_keys", [False, True])
@pytest.mark.parametrize("Hq,Hkv,D,bs,dtype", [(4, 2, 64, 32, torch.bfloat16), (3, 3, 128, 16, torch.float16),
                                               (2, 2, 64, 16, torch.bfloat16), (4, 1, 128, 32, torch.float16)])
def test_packed_fine_blocks_from_any_position(Hq, Hkv, D, bs, dtype, many_keys):
    """Decode tokens and chunks of 16- and 32-token patterns that do not start on a 64-token boundary: a tile's
    sub-blocks then lie in two rows of the coarsened pattern, the last of them behind its end."""
    S = 5120
    pk = dict(block_size=bs, local_blocks=2, vert_stride=3, num_kv_heads=Hkv)
    starts = [0, bs, 64 - bs, 64, 3 * bs, 64 + bs, 5 * bs, 7 * bs] + [4096 + bs] * (16 if many_keys else 0)
    q_lens = [1, 64, 130, 1, 63, 1, bs, 200] + [1] * (16 if many_keys else 0)
    k_lens = [a + n for a, n in zip(starts, q_lens)]
    q_lens, k_lens = q_lens + [1, 1, 64], k_lens + [48, 333, S]
    assert (sum(k_lens) > 65536) == many_keys
    cu_q, cu_k = (torch.tensor(np.cumsum([0] + n), dtype=torch.int32) for n in (q_lens, k_lens))
    q, k, v = seeded_qkv(107, (sum(q_lens), Hq, D), (sum(k_lens), Hkv, D), dtype)
    ref, ref_lse = O.varlen_attention(q.float(), k.float(), v.float(), cu_k, O.block_mask(Hq, S, **pk), bs, cu_seqlens_q=cu_q)
    mod = _module(Hq, S, pk, impl="sm100")
    with torch.no_grad():
        out, lse = mod(q.cuda(), k.cuda(), v.cuda(), cu_seqlen_k=cu_k.cuda(), cu_seqlen_q=cu_q.cuda(), return_lse=True)
    assert_out_close(out, ref)
    assert_lse_close(lse, ref_lse)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Hq,Hkv,D", [(4, 1, 128), (8, 1, 64), (12, 1, 128), (16, 1, 64)])
def test_decode_leaves_an_infinity_in_v_one(Hq, Hkv, D, dtype):
    """+-inf in V gives +-inf in that column of the output, not NaN: no term of a weight above 0 may be 0 (q of zeros:
    equal weights, exact in 16 bits) or have the other sign; the other columns are not touched."""
    bs, S, lens = 64, 512, [512, 100, 64]
    pk = dict(block_size=bs, local_blocks=8, vert_stride=4, num_kv_heads=Hkv)
    q, k, v = seeded_qkv(109, (3, 1, Hq, D), (3, S, Hkv, D), dtype)
    q[2] = 0
    left = torch.tensor([S - n for n in lens], dtype=torch.int32)
    ref, _ = O.decode_attention(q.float(), k.float(), v.float(), O.block_mask(Hq, S, **pk), bs, left_paddings=left)
    v[:, S - 50, :, 3], v[:, S - 7, :, D - 1] = float("inf"), float("-inf")
    with torch.no_grad():
        out = _module(Hq, S, pk, seq_dim=1)(q.cuda(), k.cuda(), v.cuda(), left_paddings=left.cuda()).cpu()
    assert (out[..., 3] == float("inf")).all() and (out[..., D - 1] == float("-inf")).all()
    keep = [c for c in range(D) if c not in (3, D - 1)]
    assert_out_close(out[..., keep], ref[..., keep])


@pytest.mark.parametrize("D,bs,dtype", [(64, 64, torch.bfloat16), (128, 64, torch.float16), (64, 32, torch.float16)])
def test_packed_batch_with_more_than_64k_keys_leaves_an_infinity_in_v_one(D, bs, dtype):
    Hq, Hkv, S, n_seq = 2, 1, 4096, 17
    pk = dict(block_size=bs, local_blocks=256 // bs, vert_stride=5, num_kv_heads=Hkv)
    q_lens = [1 if i % 3 == 0 else 67 for i in range(n_seq)]
    k_lens = [3840 + n for n in q_lens]
    cu_q, cu_k = (torch.tensor(np.cumsum([0] + n), dtype=torch.int32) for n in (q_lens, k_lens))
    q, k, v = seeded_qkv(111, (sum(q_lens), Hq, D), (sum(k_lens), Hkv, D), dtype)
    q[:40] = 0
    mod = _module(Hq, S, pk, impl="sm100")

    def call():
        with torch.no_grad():
            return mod(q.cuda(), k.cuda(), v.cuda(), cu_seqlen_k=cu_k.cuda(), cu_seqlen_q=cu_q.cuda()).cpu()
    ref = call()
    first = cu_k[:-1].long() + 3840             # every query of a sequence attends its first one's key
    v[first, :, 3], v[first, :, D - 1] = float("inf"), float("-inf")
    out = call()
    assert (out[..., 3] == float("inf")).all() and (out[..., D - 1] == float("-inf")).all()
    assert torch.equal(out[..., 4:D - 1], ref[..., 4:D - 1])
