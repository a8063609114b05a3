"""The tcgen05 matvec where it can go wrong: a K range that ends inside a stage, group counts whose scale rows no tensor copy can
fetch, one chunk only, column blocks on both sides of every width, bf16 rows, and ring slots that change hands between warps
(results have to repeat bit for bit however the warps interleave)."""
import pytest
import torch

from helpers import cabi, quant_ops, rel_l2, synth, to_dev
from oracle import quant_ops as oq

pytestmark = pytest.mark.gpu


def _ref(bits):
    return oq.reference_q4_matvec_decode if bits == 4 else oq.reference_q8_matvec_decode


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("B,N,K,G", [(5, 128, 128, 64), (6, 300, 1152, 128), (16, 129, 2592, 32), (17, 257, 1056, 32), (33, 64, 4096, 64), (65, 500, 640, 64),
                                     (128, 200, 1024, 64), (129, 333, 512, 64), (256, 130, 1536, 32)])
@pytest.mark.parametrize("dtype,tol", [(torch.float16, 1e-3), (torch.bfloat16, 6e-3)])
def test_shapes(cuda, bits, B, N, K, G, dtype, tol):
    w, s, z = synth.quantized_weight(N, K, bits, G, seed=N + K)
    x = synth.activations((B, K), 7, "cpu", dtype)
    for zeros in (z, None):
        want = _ref(bits)(x, w, s, zeros, group_size=G)
        got = quant_ops.matvec_rows(bits, *to_dev(cuda, x, w, s, zeros), G)
        assert rel_l2(got, want) <= tol
    assert cabi.device_status() == 0


@pytest.mark.parametrize("B,N,K,G", [(8, 4096, 4096, 64), (40, 3000, 4096, 32), (130, 14336, 2048, 64), (200, 9000, 1024, 128)])
@pytest.mark.parametrize("bits", [4, 8])
def test_results_repeat(cuda, bits, B, N, K, G):
    g, u = (tuple(t.to(cuda) for t in synth.quantized_weight(N, K, bits, G, seed=i)) for i in (1, 2))
    x = synth.activations((B, K), 3, cuda)
    plain = quant_ops.matvec_rows(bits, x, *g, G)
    pair = quant_ops.q4_gate_up_matvec_tiled if bits == 4 else quant_ops.q8_gate_up_matvec_tiled
    both = pair(x, g[0], u[0], g[1], u[1], g[2], u[2], group_size=G)
    other = torch.empty(64 << 20, dtype=torch.uint8, device=cuda)
    for i in range(20):
        if i % 4 == 0:
            other.zero_()                                  # the next launch starts from a cold cache
        assert torch.equal(quant_ops.matvec_rows(bits, x, *g, G), plain)
        assert all(torch.equal(a, b) for a, b in zip(pair(x, g[0], u[0], g[1], u[1], g[2], u[2], group_size=G), both))
    assert cabi.device_status() == 0


@pytest.mark.parametrize("B,N,K", [(5, 20480, 640), (6, 20000, 896), (40, 19300, 2944), (1024, 4096, 5504)])
def test_odd_chunk_counts_over_several_items(cuda, B, N, K):
    """q8 matrices with an odd number of 128-k chunks and more work items than SMs: the two MMA warps change places from one
    item to the next."""
    w, s, z = synth.quantized_weight(N, K, 8, 64, seed=K)
    x = synth.activations((B, K), 8)
    want = _ref(8)(x, w, s, z, group_size=64)
    args = to_dev(cuda, x, w, s, z)
    got = quant_ops.matvec_rows(8, *args, 64)
    assert rel_l2(got, want) <= 1e-3
    for _ in range(5):
        assert torch.equal(quant_ops.matvec_rows(8, *args, 64), got)
    assert cabi.device_status() == 0


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("B,N,K,G,dtype", [(9, 130, 1024, 64, torch.bfloat16), (40, 257, 4096, 128, torch.bfloat16), (130, 200, 1024, 32, torch.bfloat16),
                                           (6, 10000, 4096, 64, torch.bfloat16), (9, 130, 1152, 128, torch.float16), (17, 300, 2592, 32, torch.float16),
                                           (150, 140, 1088, 64, torch.float16)])
def test_weights_are_not_rounded(cuda, bits, B, N, K, G, dtype):
    """bf16 rows, and scale rows that no tensor copy can fetch: every result is the difference of two weights whose scales are
    neighbouring halves, 2^-10 of a weight or less, so that a weight rounded to fp16 (2^-12 of it) would show as a quarter of the result."""
    g = torch.Generator().manual_seed(B)
    codes = torch.randint(1, 16 if bits == 4 else 256, (N, 1), generator=g, dtype=torch.int32).expand(N, K).to(torch.uint8)
    w = quant_ops.pack_q4(codes) if bits == 4 else codes.contiguous()
    groups = K // G
    base = (torch.rand((N, 1), generator=g) * 0.5 + 1.0).half()
    step = torch.arange(groups) % 2                                 # scale s, s + ulp, s, ...
    scales = (base.view(torch.int16) + step.to(torch.int16)).view(torch.float16).contiguous()
    x = torch.zeros((B, K), dtype=dtype)
    for b in range(B):                                              # one element of an odd group against one of the group before it
        first = 2 * (b % (groups // 2))
        x[b, (first + 1) * G + b % G], x[b, first * G + (7 * b) % G] = 1.0, -1.0
    want = codes[:, 0].double() * (scales[:, 1].double() - scales[:, 0].double())
    for gate_up in (False, True):
        args = to_dev(cuda, x, w, scales)
        if gate_up:
            out = quant_ops.gate_up_rows(bits, args[0], args[1], args[1], args[2], args[2], None, None, G)
            got = torch.stack([out["gate"], out["up"]]).cpu()
        else:
            got = quant_ops.matvec_rows(bits, *args, None, G).cpu()[None]
        err = (got.double() - want).abs() / want
        assert err.max() <= (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8)      # twice the rounding of the result
    assert cabi.device_status() == 0


@pytest.mark.parametrize("bits,B,N,K,G", [(4, 12, 4561, 1280, 128), (8, 24, 1000, 1088, 64), (4, 6, 700, 2592, 32)])
def test_error_is_the_rounding_of_the_result(cuda, bits, B, N, K, G):
    """Against fp64, fractional zero points among them: one rounding to fp16 is 2^-12 of a value at most (2.9e-4 in the norm with
    weights rounded to fp16)."""
    w, s, z = synth.quantized_weight(N, K, bits, G, seed=N)
    x = synth.activations((B, K), 3)
    q = (torch.stack([w & 15, w >> 4], -1).reshape(N, K) if bits == 4 else w).double()
    want = x.double() @ ((q - z.double().repeat_interleave(G, 1)) * s.double().repeat_interleave(G, 1)).T
    assert rel_l2(quant_ops.matvec_rows(bits, *to_dev(cuda, x, w, s, z), G), want) <= 2.0 ** -12


@pytest.mark.parametrize("rows", [5, 8, 33])
@pytest.mark.parametrize("dtype,tol", [(torch.float16, 1e-3), (torch.bfloat16, 6e-3)])
@pytest.mark.parametrize("wide", [False, True])
def test_norm_prologue_without_a_buffer(cuda, rows, dtype, tol, wide):
    """A norm in front of the matvec with no buffer for its rows: with scratch the same launches and bits as with the buffer; with scratch
    too small for it, or none, the fused kernels and the same result up to rounding."""
    lib = cabi.load()
    N, K, G = (9600, 2560, 64) if wide else (384, 1024, 64)
    w, s, z = (t.to(cuda) for t in synth.quantized_weight(N, K, 4, G, seed=9))
    x, res = (synth.activations((rows, K), i, cuda, dtype) for i in (1, 2))
    nw = (torch.rand(K, generator=torch.Generator().manual_seed(3)) + 0.5).half().to(cuda)
    code = cabi.dtype_code(dtype)
    need = lib.b200q_norm_scratch_bytes(rows, K, code)
    assert need >= rows * K * 2 and lib.b200q_norm_scratch_bytes(4, K, code) == 0

    def call(gate_up, normed, scratch):
        out, zs = torch.empty((rows, N), dtype=dtype, device=cuda), torch.empty_like(x)
        lib.b200q_scratch_next(cabi.ptr(scratch), 0 if scratch is None else scratch.numel())
        if gate_up:
            rc = lib.b200q_gate_up_swiglu(4, x.data_ptr(), w.data_ptr(), w.data_ptr(), s.data_ptr(), s.data_ptr(), z.data_ptr(), z.data_ptr(), None, None,
                                          out.data_ptr(), res.data_ptr(), nw.data_ptr(), cabi.F16, 1e-5, zs.data_ptr(), cabi.ptr(normed), rows, N, K, G,
                                          code, cabi.F16, cabi.stream())
        else:
            rc = lib.b200q_norm_qmatvec(4, x.data_ptr(), res.data_ptr(), nw.data_ptr(), cabi.F16, 1e-5, zs.data_ptr(), cabi.ptr(normed), w.data_ptr(),
                                        s.data_ptr(), z.data_ptr(), None, out.data_ptr(), rows, N, K, G, code, cabi.F16, cabi.stream())
        assert rc == 0
        return out, zs

    new = lambda n: torch.empty(n, dtype=torch.uint8, device=cuda)
    for gate_up in (False, True):
        want = call(gate_up, torch.empty_like(x), new(need))
        got = call(gate_up, None, new(need))
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        for scratch in (None, new(lib.b200q_scratch_bytes(rows, K, code) or 256)):
            got = call(gate_up, None, scratch)
            assert rel_l2(got[0], want[0]) <= 2 * tol and torch.equal(got[1], want[1])
    assert cabi.device_status() == 0
