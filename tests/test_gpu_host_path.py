"""The operators' native call path against their Python bodies: the same launches, bit for bit, on the ordinary arguments;
None (the Python body takes the call) on everything else."""
import ctypes

import pytest
import torch

from helpers import cabi, mlp_ops, pq_ops, quant_ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,shape,dtype", [(4, (1, 256), torch.float16), (8, (3, 1, 512), torch.bfloat16), (4, (33, 192), torch.float16)])
def test_matvec_equals_python_body(cuda, bits, shape, dtype):
    K = shape[-1]
    w, s, z = (t.to(cuda) for t in synth.quantized_weight(130, K, bits, 32, seed=3))
    x = synth.activations(shape, 4, cuda, dtype)
    host = cabi.host()
    for backend in ("cuda", "auto", "metal_tiled"):
        got = host.matvec(bits, x, w, s, z, 32, backend)
        assert got is not None and torch.equal(got, quant_ops.matvec_rows(bits, x.reshape(-1, K), w, s, z, 32))
    # calls for the Python body: to convert, to refuse, or to reject with its message
    assert host.matvec(bits, x, w, s.to(torch.float64), z, 32, "cuda") is None
    assert host.matvec(bits, x, w, s, z[:, :1], 32, "cuda") is None
    assert host.matvec(bits, x, w.cpu(), s, z, 32, "cuda") is None
    assert host.matvec(bits, x.float(), w, s, z, 32, "cuda") is None
    assert host.matvec(bits, x, w, s, z, 32, "reference") is None


@pytest.mark.parametrize("rows", [1, 4, 5, 40])
def test_mlp_block_equals_python_body(cuda, rows):
    D, inter, G = 256, 448, 64
    mats = [tuple(t.to(cuda) for t in synth.quantized_weight(n, k, 4, G, seed=n + k)) for n, k in ((inter, D), (inter, D), (D, inter))]
    (gw, gs, gz), (uw, us, uz), (dw, ds, dz) = mats
    x, r = (synth.activations((1, rows, D), s, cuda) for s in (5, 6))
    nw = torch.ones(D, dtype=torch.float16, device=cuda)
    got = cabi.host().mlp_block(x, r, nw, gw, gs, gz, uw, us, uz, dw, ds, dz, 4, G, 1e-5)
    assert got is not None
    want = mlp_ops.quantized_mlp_block(x, r, nw, gw, gs, uw, us, dw, ds, gate_zeros=gz, up_zeros=uz, down_zeros=dz, bits=4,
                                       group_size=G, backend_preset="tiled")      # the preset that stays in the Python body
    assert torch.equal(got, want)


@pytest.mark.parametrize("window", [0, 20])
@pytest.mark.parametrize("batch", [1, 9])
def test_paged_attention_equals_python_body(cuda, batch, window):
    case = synth.paged_kv_case(batch, 8, 128, 16, num_pages=400, min_len=1, max_len=300, bits=8, group_size=32, seed=2)
    cache = pq_ops.PagedQuantizedKVCache(**{k: (v.to(cuda) if torch.is_tensor(v) else v) for k, v in case.items()})
    q = synth.activations((batch, 1, 32, 128), 8, cuda)
    got = cabi.host().paged_attention(q, cache, None, 4, window)
    want = pq_ops.paged_attention_launch(q.reshape(batch, 32, 128), cache, 128 ** -0.5, sink_tokens=4, window_size=window)
    assert got is not None and torch.equal(got.reshape(want.shape), want)
    cache.lengths = cache.lengths.to(torch.int64)
    assert cabi.host().paged_attention(q, cache, None, 4, window) is None


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("pages,D,G,dtype", [(1, 128, 32, torch.float16), (5, 128, 64, torch.bfloat16), (67, 64, 8, torch.float16),
                                             (3, 512, 256, torch.float16), (2, 24, 8, torch.bfloat16), (2, 48, 32, torch.float16)])
def test_quantised_pages_equal_python_body(cuda, bits, pages, D, G, dtype):
    """K and V pages through the 16-byte kernels and back: codes and scales of the oracle's rule bit for bit, for values on
    and next to the ties of the rounding, zero groups and outliers; the last shape (a short last group) takes the general ones."""
    k, v = (synth.activations((pages, 16, 3, D), s, "cpu", dtype) for s in (21, 22))
    k.view(-1)[:G] = 0.0
    limit = 127 if bits == 8 else 7
    v.view(-1)[:G] = ((torch.arange(G) % (2 * limit)).float() - limit + 0.5).to(dtype)      # scale near 1: quotients at ties
    v.view(-1)[0] = float(limit)
    v.view(-1)[-1] = 3.0e4
    bt, ln = torch.zeros((1, 1), dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    got = pq_ops.quantize_kv_pages(k.to(cuda), v.to(cuda), bt, ln, pq_ops.PagedQuantizedKVConfig(bits=bits, group_size=G))
    for pages_t, codes, scales in ((k, got.k_pages_q, got.k_scales), (v, got.v_pages_q, got.v_scales)):
        oc, osc = synth.quantize_kv_symmetric(pages_t, bits, G)
        assert torch.equal(codes.cpu(), oc) and torch.equal(scales.cpu(), osc)
    kd, vd = pq_ops.dequantize_kv_pages(got)
    off = 128.0 if bits == 8 else 8.0
    for out, codes, scales in ((kd, got.k_pages_q, got.k_scales), (vd, got.v_pages_q, got.v_scales)):
        rows = out.numel() // D
        s = scales.reshape(rows, -1).abs()
        ref = quant_ops.dequant_codes(bits, codes.reshape(rows, -1), s, torch.full_like(s, off), rows, D, G, torch.float16)
        assert torch.equal(out.reshape(rows, D), ref)


@pytest.mark.parametrize("code,falls_through", [(-2, True), (-4, True), (-3, False), (-1, False)])
def test_plain_attention_falls_through_only_where_nothing_was_launched(cuda, code, falls_through):
    """The entry point that reports on the lengths fails with ``code``: after a failed launch its kernel may be under way, so the
    general one must not be launched on the same workspace.  The entry points are stand-ins: no kernel runs."""
    lib, host, calls = cabi.load(), cabi.host(), []

    def stand_in(name, result):
        restype, argtypes = cabi.SIGNATURES[name]
        return ctypes.CFUNCTYPE(restype, *argtypes)(lambda *args: calls.append(name) or result)

    fakes = {"b200q_paged_fp16_gqa_decode_checked": stand_in("b200q_paged_fp16_gqa_decode_checked", code),
             "b200q_paged_fp16_gqa_decode": stand_in("b200q_paged_fp16_gqa_decode", -2)}
    table = {name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in cabi.SIGNATURES}
    pages = synth.activations((4, 16, 8, 128), 1, cuda)
    q = synth.activations((1, 1, 8, 128), 2, cuda)
    bt, ln = torch.arange(4, dtype=torch.int32, device=cuda).reshape(1, 4), torch.tensor([50], dtype=torch.int32, device=cuda)
    host.bind({**table, **{name: ctypes.cast(fn, ctypes.c_void_p).value for name, fn in fakes.items()}})
    try:
        assert host.plain_attention(q, pages, pages, bt, ln, None) is None
    finally:
        host.bind(table)
    assert calls == list(fakes)[:2 if falls_through else 1]
    assert host.plain_attention(q, pages, pages, bt, ln, None) is not None
