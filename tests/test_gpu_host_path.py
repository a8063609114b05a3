"""The operators' native call path against their Python bodies: the same launches, bit for bit, on the ordinary arguments;
None (the Python body takes the call) on everything else."""
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
