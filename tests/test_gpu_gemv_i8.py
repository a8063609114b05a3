"""The integer tensor-core matvec (one to four rows) against the oracle: unit, tile and group remainders, both row types, zero
points absent, the fused norm and residual, values that stress its fixed-point activations, and row shards bit for bit."""
import pytest
import torch

from helpers import cabi, mlp_ops, quant_ops, rel_l2, synth, to_dev
from oracle import quant_ops as oq

pytestmark = pytest.mark.gpu


def _ref(bits):
    return oq.reference_q4_matvec_decode if bits == 4 else oq.reference_q8_matvec_decode


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("B,N,K,G", [(1, 1, 64, 32), (2, 17, 64, 64), (3, 333, 2592, 32), (4, 150, 640, 64), (1, 4097, 1024, 128),
                                     (2, 600, 4096, 64), (4, 260, 4096, 32), (1, 64, 14336, 64), (1, 40000, 128, 64), (3, 2000, 384, 128)])
def test_shapes(cuda, bits, B, N, K, G):
    w, s, z = synth.quantized_weight(N, K, bits, G, seed=N + K)
    for dtype, tol in ((torch.float16, 1e-3), (torch.bfloat16, 6e-3)):
        x = synth.activations((B, K), 7, "cpu", dtype)
        for zeros in (z, None):
            want = _ref(bits)(x, w, s, zeros, group_size=G)
            got = quant_ops.matvec_rows(bits, *to_dev(cuda, x, w, s, zeros), G)
            assert rel_l2(got, want) <= tol
    assert cabi.device_status() == 0


def test_outliers_and_empty_groups(cuda):
    """Groups of zeros, an outlier of 2^14 beside small values, and the smallest normal halves."""
    w, s, z = synth.quantized_weight(256, 1024, 4, 64, seed=3)
    x = synth.activations((2, 1024), 9)
    x[0, :64] = 0
    x[0, 70] = 16384.0
    x[1] *= 2.0 ** -14
    want = _ref(4)(x, w, s, z, group_size=64)
    got = quant_ops.matvec_rows(4, *to_dev(cuda, x, w, s, z), 64)
    assert rel_l2(got[:1], want[:1]) <= 1e-3 and rel_l2(got[1:], want[1:]) <= 6e-3      # the second row's results are subnormal halves


@pytest.mark.parametrize("bits,G", [(8, 128), (8, 32), (4, 128), (4, 64)])
@pytest.mark.parametrize("rows", [1, 2, 4])
def test_largest_digit_sums(cuda, bits, G, rows):
    """Codes and activations at their limits of one sign: the digit sums of a group come within 0.4 % of the range that the integers added
    to a float's bits have.  fp32 sums of equal terms: error below 2^-11 of the result from its rounding to fp16."""
    N, K = 50, 4 * G + 32 * (G == 32)
    codes = torch.full((N, K * bits // 8), 255, dtype=torch.uint8)
    scales = torch.full((N, K // G), 2.0 ** -12, dtype=torch.float16)
    zeros = torch.full((N, K // G), 3.0, dtype=torch.float16)
    for value in (-1.0, 0.99951171875):
        x = torch.full((rows, K), value, dtype=torch.float16)
        want = torch.full((rows, N), K * value * (2 ** bits - 1 - 3) * 2.0 ** -12, dtype=torch.float64)
        got = quant_ops.matvec_rows(bits, *to_dev(cuda, x, codes, scales, zeros), G)
        assert rel_l2(got, want) <= 2.0 ** -11


@pytest.mark.parametrize("bits,G", [(4, 32), (4, 64), (4, 128), (8, 32), (8, 64), (8, 128)])
@pytest.mark.parametrize("units,tail", [(1, 1), (1, 2), (2, 4), (2, 8), (3, 4), (7, 6), (22, 2), (22, 7)])
def test_rows_that_end_inside_a_unit(cuda, bits, G, units, tail):
    """Rows of scales that start at multiples of 2, 4, 8 or 16 bytes: the same bits as rows that are padded to whole units, whose added
    activations are zero and whose codes and scales are anything."""
    per_unit = 2048 // bits // G
    groups = (units - 1) * per_unit + min(tail, per_unit - 1)
    K, Kp, N = groups * G, units * per_unit * G, 148 * 34 + 11 if units <= 7 else 148 * 20 + 5
    w, s, z = (t.to(cuda) for t in synth.quantized_weight(N, Kp, bits, G, seed=units + G))
    x = torch.zeros((4, Kp), dtype=torch.float16, device=cuda)
    x[:, :K] = synth.activations((4, K), 3, cuda)
    for rows in (1, 2, 4) if units <= 7 else (1, 2):      # (four rows of 22 units can exceed an SM's shared memory: another kernel)
        for zeros in (z, None):
            want = quant_ops.matvec_rows(bits, x[:rows].contiguous(), w, s, zeros, G)
            got = quant_ops.matvec_rows(bits, x[:rows, :K].contiguous(), w[:, :K * bits // 8].contiguous(), s[:, :groups].contiguous(),
                                        None if zeros is None else zeros[:, :groups].contiguous(), G)
            assert torch.equal(got, want)
    assert cabi.device_status() == 0


@pytest.mark.parametrize("bits,K,G,N", [(4, 14336, 64, 1000), (4, 14336, 32, 5), (8, 7200, 32, 4101), (4, 11008, 128, 700), (8, 14336, 64, 9)])
def test_long_rows_by_pairs_of_ctas(cuda, bits, K, G, N):
    """Rows that two CTAs share, also for gate/up; two and three rows, which may have a CTA to themselves, give the same bits as among four,
    whose digits do not fit one CTA (but for the rows of 7200).  Against the oracle: fp32 sums rounded to fp16, below 2^-11."""
    w, s, z = synth.quantized_weight(N, K, bits, G, seed=K + N)
    x = synth.activations((4, K), 2, "cpu")
    dev = to_dev(cuda, x, w, s, z)
    got = quant_ops.matvec_rows(bits, *dev, G)
    assert rel_l2(got, _ref(bits)(x, w, s, z, group_size=G)) <= 1e-3
    for rows in (2, 3):
        assert torch.equal(quant_ops.matvec_rows(bits, dev[0][:rows].contiguous(), *dev[1:], G), got[:rows])
    assert rel_l2(quant_ops.matvec_rows(bits, dev[0][:1].contiguous(), *dev[1:], G), got[:1]) <= 2.0 ** -10
    both = quant_ops.gate_up_rows(bits, dev[0], dev[1], dev[1], dev[2], dev[2], dev[3], dev[3], G, want_gate_up=True, want_act=False)
    assert torch.equal(both["gate"], got) and torch.equal(both["up"], got)
    assert cabi.device_status() == 0


@pytest.mark.parametrize("power", [120, 100, -60, -100])
def test_bf16_rows_near_both_ends_of_the_range(cuda, power):
    """bf16 rows times a power of two give the same results times that power, bit for bit, as long as these are in range."""
    w, s, z = synth.quantized_weight(70, 256, 4, 64, seed=8)
    x = synth.activations((2, 256), 9, "cpu", torch.bfloat16)
    s = (s.float() * 2.0 ** -6).to(torch.float16)
    near = quant_ops.matvec_rows(4, *to_dev(cuda, x, w, s, z), 64)
    far = quant_ops.matvec_rows(4, *to_dev(cuda, (x.float() * 2.0 ** power).to(torch.bfloat16), w, s, z), 64)
    assert torch.equal(far.float() * 2.0 ** -power, near.float())


def _exact(x, w, s, z, bits, G):
    N, K = w.shape[0], x.shape[1]
    codes = (torch.stack((w & 15, w >> 4), -1).reshape(N, K) if bits == 4 else w).double()
    dense = (codes.reshape(N, K // G, G) - z.double()[..., None]) * s.double()[..., None]
    return x.double() @ dense.reshape(N, K).T


@pytest.mark.parametrize("bits,K", [(4, 256), (8, 14336)])
@pytest.mark.parametrize("powers", [(-104, -23), (-110, -17), (-90, -24)])
def test_small_bf16_rows_with_small_scales(cuda, bits, K, powers):
    """Results near the lower end of bf16's normal range are right to their own rounding (2^-9) and that of the rows to fixed point (steps of
    2^-120, 2^-10 of the smallest rows' values here, independent of one another: 2^-11 of the result)."""
    w, s, z = synth.quantized_weight(70, K, bits, 64, seed=8)
    s = torch.full_like(s, 2.0 ** powers[1], dtype=torch.float16)
    x = (synth.activations((4, K), 9, "cpu", torch.bfloat16).double() * 2.0 ** powers[0]).to(torch.bfloat16)
    for rows in (1, 2, 4):
        got = quant_ops.matvec_rows(bits, *to_dev(cuda, x[:rows].contiguous(), w, s, z), 64)
        assert rel_l2(got, _exact(x[:rows], w, s, z, bits, 64)) <= 2.0 ** -9 + 2.0 ** -11


@pytest.mark.parametrize("bits,K", [(4, 256), (4, 14336), (8, 14336)])
def test_large_and_small_bf16_rows_together(cuda, bits, K):
    """Rows near both ends of bf16's range, and one whose values lie near both, in one call: each is right to its own rounding, and the
    same bits as by itself."""
    w, s, z = synth.quantized_weight(70, K, bits, 64, seed=11)
    s = torch.full_like(s, 2.0 ** -20, dtype=torch.float16)
    x = synth.activations((4, K), 12, "cpu", torch.bfloat16).double()
    x[0] *= 2.0 ** 120                        # the sum of a group (at most 64 values of 2^123) stays finite in fp32
    x[1] *= 2.0 ** -104
    x[2, :K - 64] *= 2.0 ** 60
    x[2, K - 64:] *= 2.0 ** 110
    x = x.to(torch.bfloat16)
    dev = to_dev(cuda, x, w, s, z)
    got = quant_ops.matvec_rows(bits, *dev, 64)
    want = _exact(x, w, s, z, bits, 64)
    for row in range(4):
        assert rel_l2(got[row], want[row]) <= 2.0 ** -9 + 2.0 ** -11
        pair = quant_ops.matvec_rows(bits, dev[0][[row, row]].contiguous(), *dev[1:], 64)
        assert torch.equal(pair[0], got[row]) and torch.equal(pair[1], got[row])


@pytest.mark.parametrize("rows", [1, 2, 4])
@pytest.mark.parametrize("lo,hi", [(0, 96), (96, 333), (5, 6)])
def test_row_shards_reproduce_the_unsharded_rows(cuda, rows, lo, hi):
    w, s, z = (t.to(cuda) for t in synth.quantized_weight(333, 1024, 4, 64, seed=5))
    x = synth.activations((rows, 1024), 6, cuda)
    full = quant_ops.matvec_rows(4, x, w, s, z, 64)
    part = quant_ops.matvec_rows(4, x, w[lo:hi].contiguous(), s[lo:hi].contiguous(), z[lo:hi].contiguous(), 64)
    assert torch.equal(part, full[:, lo:hi])
