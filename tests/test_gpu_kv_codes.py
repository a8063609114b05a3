"""The 16-byte KV quantiser where its reciprocal could go wrong: exact ties, tiny and large groups, and values that are not finite
(their warps divide).  Codes and scales have to be those of the rule in fp32, byte for byte."""
import pytest
import torch

from helpers import pq_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits,G", [(4, 32), (8, 32), (8, 128), (4, 8)])
def test_codes(cuda, dtype, bits, G):
    g = torch.Generator().manual_seed(bits + G)
    limit, offset = (127, 128) if bits == 8 else (7, 8)
    x = torch.randn((9, 16, 3, 128), generator=g)
    x[1] = torch.randint(-2 * limit, 2 * limit + 1, x[1].shape, generator=g).float() / 2      # many quotients lie on a tie
    x[2] *= 1e-6
    x[3] *= 3e4
    x[4] = 0
    x[5, 3, 1, 7], x[6, 0, 2, 100] = float("inf"), -float("inf")
    x = x.to(dtype)
    table, lengths = torch.arange(9, dtype=torch.int32).reshape(1, -1), torch.tensor([144], dtype=torch.int32)
    cache = pq_ops.quantize_kv_pages(x.to(cuda), x.to(cuda), table.to(cuda), lengths.to(cuda), pq_ops.PagedQuantizedKVConfig(bits=bits, group_size=G))
    v = x.float().reshape(-1, G)
    scale = torch.clamp(v.abs().amax(-1, keepdim=True), min=1e-8) / torch.tensor(float(limit))
    want = torch.clamp(torch.nan_to_num(torch.round(v / scale), nan=-float(limit)), -limit, limit).to(torch.int32) + offset
    for codes, scales in ((cache.k_pages_q, cache.k_scales), (cache.v_pages_q, cache.v_scales)):
        c = codes.cpu().to(torch.int32)
        if bits == 4:
            c = torch.stack([c & 15, c >> 4], -1)
        assert torch.equal(c.reshape(-1, G), want)
        assert torch.equal(scales.cpu().reshape(-1, 1), scale.half())
