"""4-bit keys whose scales lie at the ends of bfloat16's range (the quotients then keep their residual correction) beside ordinary ones
in the same call, bit for bit against the CPU oracle."""

import pytest
import torch

from oracle import group_format as gf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-31, -29, 0, 29, 31, 37])
def test_scales_at_the_ends_of_the_range(exponent):
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(100 + exponent)
    x = torch.rand(1, 2, 96, 128, generator=g)
    x[..., ::2] *= 10.0 ** exponent
    x = x.to(torch.bfloat16)
    code, scale, mn = ops.pack_k_per_channel(x.cuda(), 32, 4)
    ref = gf.quantize_and_pack_last_dim(x.transpose(2, 3).contiguous(), 32, 4)
    assert torch.equal(code.cpu(), ref[0])
    assert torch.equal(scale.cpu().view(torch.int16), ref[1].view(torch.int16).view(scale.shape))
    assert torch.equal(mn.cpu().view(torch.int16), ref[2].view(torch.int16).view(mn.shape))
