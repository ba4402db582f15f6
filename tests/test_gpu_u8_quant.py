"""Quantize + encode of a span in one launch against the CPU oracle, bit for bit: every cluster size, slices of uneven length,
a single token, degenerate channels (which take the per-element arithmetic), thresholds close to zero, both data types."""

import pytest
import torch

from oracle import calibquant_format as cqf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits,clip", [(1, 0.5), (2, 1), (4, 1)])
@pytest.mark.parametrize("B,T,H,constant", [(1, 1, 1, False), (1, 127, 2, False), (2, 130, 8, True), (1, 259, 3, False), (1, 1283, 8, False),
                                            (1, 2050, 2, False), (40, 96, 8, False)])
def test_quant_encode(dtype, bits, clip, B, T, H, constant):
    from calibquant_b200 import calibquant as cq
    g = torch.Generator().manual_seed(T + bits)
    x = torch.randn(B, T, H + 1, 128, generator=g) * torch.exp(torch.randn(128, generator=g)) + torch.randn(128, generator=g)
    if T > 1:
        x[:, :, :, 5] = x[:, :, :, 5].abs() * 1e-3      # one-sided channels: extremes next to zero
    if constant:
        x[0, :, 0, 7] = 1.5
    x = x.to(dtype)[:, :, :H]
    enc, s, z = cq.quant_encode(x.cuda(), bits, scale=clip)
    ref, rs, rz = cqf.quant(x, bits, per_channel=True, scale=clip, post_scale=True)
    assert torch.equal(torch.nan_to_num(s.cpu().float()), torch.nan_to_num(rs.float()))
    assert torch.equal(torch.nan_to_num(z.cpu().float()), torch.nan_to_num(rz.float()))
    good = torch.isfinite(ref.float())                  # a constant channel has scale 0 and no codes
    assert T == 1 or constant or bool(good.all())
    mine = cqf.decode_bytes(enc.cpu(), bits).transpose(1, 2)
    assert torch.equal(mine[good].to(torch.int64), ref[good].to(torch.int64))


@pytest.mark.parametrize("B,T,H", [(1, 8300, 1), (2, 9001, 2), (1, 8192, 8)])
def test_long_spans_of_few_heads_at_four_bits(B, T, H):
    """Spans that the separate launches take: bytes, scales and zero points of the oracle."""
    from calibquant_b200 import calibquant as cq
    x = torch.randn(B, T, H, 128, generator=torch.Generator().manual_seed(T)).half()
    codes, s, z = cqf.quant(x, 4, per_channel=True, post_scale=True)
    enc, s_out, z_out = (t.cpu() for t in cq.quant_encode(x.cuda(), 4))
    assert torch.equal(enc, cqf.encode(codes.transpose(1, 2), 4, 2))
    assert torch.equal(s_out, s) and torch.equal(z_out, z)
