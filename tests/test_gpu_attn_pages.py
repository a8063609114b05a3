"""Decode attention through the page building blocks (quantised and plain pages) where they can go wrong: both layouts of the
query heads, bf16 queries, chunks of kv heads, a maximum that keeps moving, V scales far apart, and slots past the length
that hold anything at all."""
import pytest
import torch

from helpers import cabi, pq_ops, rel_l2, synth
import importlib

gqa_ops = importlib.import_module("mlx_metal_kernels_b200.ops.gqa_ops")
pytestmark = pytest.mark.gpu


def _expected(q, k, v, table, lengths):
    """softmax(q k / sqrt(D)) v in fp64 over the first lengths[b] tokens, from dequantised pages [pages, 16, Hkv, D]."""
    B, _, Hq, D = q.shape
    Hkv = k.shape[2]
    out = torch.zeros(B, 1, Hq, D, dtype=torch.float64)
    for b in range(B):
        L = int(lengths[b])
        if L == 0:
            continue
        pages = table[b, :(L + 15) // 16].long()
        kb, vb = (t[pages].reshape(-1, Hkv, D)[:L].double().repeat_interleave(Hq // Hkv, 1) for t in (k, v))
        p = torch.softmax(torch.einsum("hd,lhd->hl", q[b, 0].double(), kb) / D ** 0.5, -1)
        out[b, 0] = torch.einsum("hl,lhd->hd", p, vb)
    return out


def _table(lengths, pages, seed):
    g = torch.Generator().manual_seed(seed)
    perm = torch.randperm(pages, generator=g).to(torch.int32)
    table = torch.full((len(lengths), max(1, (max(lengths) + 15) // 16)), -1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(lengths):
        m = (n + 15) // 16
        table[b, :m] = perm[at:at + m]
        at += m
    return table


@pytest.mark.parametrize("bits,G", [(4, 32), (4, 64), (8, 32), (8, 64)])
@pytest.mark.parametrize("Hq,Hkv,lengths", [(8, 1, [1, 300, 17]), (16, 2, [16, 33]), (12, 2, [700]), (6, 3, [129, 5]), (32, 16, [40, 0, 250]),
                                            (32, 8, [2000] * 9)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_quantised_pages(cuda, bits, G, Hq, Hkv, lengths, dtype):
    pages = sum((n + 15) // 16 for n in lengths) + 3
    table, ln = _table(lengths, pages, 1), torch.tensor(lengths, dtype=torch.int32)
    k, v = (synth.activations((pages, 16, Hkv, 128), s) for s in (11, 12))
    # scores that grow along the sequence: the reference maximum moves again and again; V of one page far larger than the rest
    for b, n in enumerate(lengths):
        m = (n + 15) // 16
        k[table[b, :m].long()] *= torch.linspace(0.2, 3.0, max(m, 1))[:m].half().reshape(-1, 1, 1, 1)
        if m > 2:
            v[table[b, 2].long()] *= 200.0
    q = synth.activations((len(lengths), 1, Hq, 128), 13, "cpu", dtype)
    cache = pq_ops.quantize_kv_pages(k.to(cuda), v.to(cuda), table.to(cuda), ln.to(cuda), pq_ops.PagedQuantizedKVConfig(bits=bits, group_size=G))
    kd, vd = (t.cpu() for t in pq_ops.dequantize_kv_pages(cache))
    for b, n in enumerate(lengths):                       # scales of slots past the length: anything
        if n % 16:
            for t in (cache.k_scales, cache.v_scales):
                t[int(table[b, n // 16]), n % 16:] = float("nan")
    want = _expected(q, kd, vd, table, ln)
    tol = 2e-3 if dtype == torch.float16 else 8e-3
    for cluster in (-1, 1):
        cabi.set_tuning("attn.cluster", cluster)
        try:
            got = pq_ops.paged_quantized_kv_gqa_decode_attention(q.to(cuda), cache, backend="cuda").cpu().double()
        finally:
            cabi.set_tuning("attn.cluster", 0)
        assert (got - want).abs().max() <= tol * max(1.0, want.abs().max())
    assert cabi.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Hq,Hkv,lengths", [(8, 8, [1, 300, 17]), (16, 2, [16, 33]), (4, 1, [700, 0]), (6, 3, [129, 5]), (40, 8, [513]), (64, 16, [31] * 5)])
def test_plain_pages(cuda, dtype, Hq, Hkv, lengths):
    pages = sum((n + 15) // 16 for n in lengths) + 3
    table, ln = _table(lengths, pages, 2), torch.tensor(lengths, dtype=torch.int32)
    k, v = (synth.activations((pages, 16, Hkv, 128), s, "cpu", dtype) for s in (21, 22))
    q = synth.activations((len(lengths), 1, Hq, 128), 23, "cpu", dtype)
    want = _expected(q, k, v, table, ln)
    for b, n in enumerate(lengths):                       # slots past the length may hold anything
        if n % 16:
            for t in (k, v):
                t[int(table[b, n // 16]), n % 16:] = float("nan")
    args = [t.to(cuda) for t in (q, k, v, table, ln)]
    got = gqa_ops.paged_gqa_decode_attention(*args).cpu().double()
    assert (got - want).abs().max() <= (2e-3 if dtype == torch.float16 else 1.6e-2)
    assert cabi.host().plain_attention(*args, None) is not None
    bad = args[4].clone()
    bad[0] = 10 ** 6
    with pytest.raises(ValueError, match="positions must be in"):
        gqa_ops.paged_gqa_decode_attention(*args[:4], bad)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("cluster,size", [(-1, 0), (1, 1), (1, 2), (1, 4), (1, 8)])
@pytest.mark.parametrize("Hq,Hkv,lengths", [(8, 8, [1, 300, 17]), (4, 1, [700, 0]), (40, 8, [513]), (64, 16, [31] * 5)])
def test_plain_pages_by_both_kernels(cuda, dtype, cluster, size, Hq, Hkv, lengths):
    """Split-KV with a merge, and clusters of one to eight CTAs: walks longer than a warp's ring, warps without a page, an empty sequence."""
    pages = sum((n + 15) // 16 for n in lengths) + 3
    table, ln = _table(lengths, pages, 2), torch.tensor(lengths, dtype=torch.int32)
    k, v = (synth.activations((pages, 16, Hkv, 128), s, "cpu", dtype) for s in (21, 22))
    q = synth.activations((len(lengths), 1, Hq, 128), 23, "cpu", dtype)
    want = _expected(q, k, v, table, ln)
    cabi.set_tuning("attn.cluster", cluster)
    cabi.set_tuning("attn.cluster_size", size)
    try:
        got = gqa_ops.paged_gqa_decode_attention(*(t.to(cuda) for t in (q, k, v, table, ln))).cpu().double()
    finally:
        cabi.set_tuning("attn.cluster", 0)
        cabi.set_tuning("attn.cluster_size", 0)
    assert (got - want).abs().max() <= (2e-3 if dtype == torch.float16 else 1.6e-2)
    assert cabi.device_status() == 0


@pytest.mark.parametrize("bits,G", [(4, 32), (8, 64)])
@pytest.mark.parametrize("Hq,Hkv,lengths", [(8, 1, [1, 300, 17]), (6, 3, [129, 5]), (32, 8, [700, 0, 40]), (32, 16, [40, 0, 250])])
@pytest.mark.parametrize("shifted", ["k_scales", "v_scales", "both"])
def test_scales_aligned_to_eight_bytes(cuda, bits, G, Hq, Hkv, lengths, shifted):
    """Views of scales that start 8 bytes into a 16-byte piece give the same bits as aligned ones, in both kernels, with a page missing."""
    pages = sum((n + 15) // 16 for n in lengths) + 3
    table, ln = _table(lengths, pages, 1).to(cuda), torch.tensor(lengths, dtype=torch.int32, device=cuda)
    if table.shape[1] > 1:
        table[0, 1] = -1
    k, v = (synth.activations((pages, 16, Hkv, 128), s, cuda) for s in (31, 32))
    q = synth.activations((len(lengths), 1, Hq, 128), 33, cuda)
    cache = pq_ops.quantize_kv_pages(k, v, table, ln, pq_ops.PagedQuantizedKVConfig(bits=bits, group_size=G))
    aligned = {name: getattr(cache, name) for name in ("k_scales", "v_scales")}
    for cluster in (-1, 1):
        cabi.set_tuning("attn.cluster", cluster)
        try:
            for name in aligned:
                setattr(cache, name, aligned[name])
            want = pq_ops.paged_quantized_kv_gqa_decode_attention(q, cache, backend="cuda")
            for name in aligned:
                if shifted in (name, "both"):
                    setattr(cache, name, torch.cat([aligned[name].new_zeros(4), aligned[name].flatten()])[4:].view(aligned[name].shape))
                    assert getattr(cache, name).data_ptr() % 16 == 8
            got = pq_ops.paged_quantized_kv_gqa_decode_attention(q, cache, backend="cuda")
        finally:
            cabi.set_tuning("attn.cluster", 0)
        assert torch.equal(got, want)
    assert cabi.device_status() == 0


@pytest.mark.parametrize("bits,G", [(4, 32), (4, 64), (8, 32), (8, 64)])
@pytest.mark.parametrize("Hq,Hkv", [(8, 2), (16, 2), (5, 1)])
@pytest.mark.parametrize("kind", ["one_head", "all_heads", "two_channels", "alone_in_group"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_query_heads_with_outliers(cuda, bits, G, Hq, Hkv, kind, dtype):
    """Queries with a channel far above the rest, where K is (nearly) zero: the scores depend on elements that lie 60 to 2000 times below
    the largest.  Queries and K enter unrounded; what is left is p * scale and the result rounded once each, 2^-12 (fp16 result) or
    2^-9 (bf16) of a value at most and about 0.6 of that in the norm, so 5e-4 and 2.4e-3 bound the relative error (queries rounded
    at 2^-16 of the largest give 9e-4 and 1.9e-3 for a factor of 100, and grow with the factor)."""
    L, pages = 700, 100
    table, ln = _table([L, 33], pages, 5), torch.tensor([L, 33], dtype=torch.int32)
    k, v = (synth.activations((pages, 16, Hkv, 128), s) for s in (41, 42))
    q = synth.activations((2, 1, Hq, 128), 43, "cpu", torch.float32)
    if kind == "one_head":
        k[..., 37] = 0
        q[:, :, 1 % Hq, 37] = 100.0
    elif kind == "all_heads":
        k[..., 37] = 0
        q[..., 37] = -2000.0
    elif kind == "two_channels":
        k[..., 5] *= 1e-3
        k[..., 99] *= 1e-3
        q[..., 5], q[..., 99] = 300.0, -300.0
    else:                                                 # nothing but the outlier in the first 32 elements
        k[..., :32] *= 0.05
        q[..., :32] = 0.0
        q[..., 3] = 60.0
    q = q.to(dtype)
    cache = pq_ops.quantize_kv_pages(k.to(cuda), v.to(cuda), table.to(cuda), ln.to(cuda), pq_ops.PagedQuantizedKVConfig(bits=bits, group_size=G))
    off = 8.0 if bits == 4 else 128.0

    def exact(codes, scales):
        codes, scales = codes.cpu(), scales.cpu().double().abs()
        if bits == 4:
            codes = torch.stack([codes & 15, codes >> 4], -1).reshape(*codes.shape[:-1], 128)
        return (codes.double() - off) * scales.repeat_interleave(G, -1)

    want = _expected(q, exact(cache.k_pages_q, cache.k_scales), exact(cache.v_pages_q, cache.v_scales), table, [L, 33])
    for cluster in (-1, 1):
        cabi.set_tuning("attn.cluster", cluster)
        try:
            got = pq_ops.paged_quantized_kv_gqa_decode_attention(q.to(cuda), cache, backend="cuda")
        finally:
            cabi.set_tuning("attn.cluster", 0)
        assert rel_l2(got, want) <= (5e-4 if dtype == torch.float16 else 2.4e-3)
    assert cabi.device_status() == 0
