"""The quantized product over token counts that take the small and the large tiles of the attn.V kernel, in one process and in
either order."""

import pytest
import torch

from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2])
def test_small_and_large_tiles_in_turn(bits):
    from calibquant_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(bits)
    for K in (512, 32768, 256, 16384, 512):
        w = torch.randn(8, 32, 1, K, generator=g, device="cuda").half() * 2.0 ** -5
        code, scale, mn = ops.pack_v_per_token(torch.randn(8, 8, K, 128, generator=g, device="cuda").half(), 32, bits)
        fields = (code.unsqueeze(-1) >> (torch.arange(32 // bits, device="cuda") * bits)) & (2 ** bits - 1)
        v = fields.flatten(-2).unflatten(-1, (4, 32)).float() * scale.float().unsqueeze(-1) + mn.float().unsqueeze(-1)
        ref = w.float() @ v.flatten(-2).repeat_interleave(4, 1)
        assert rel_l2(ops.qbmm(32, w, code, scale, mn, bits), ref) <= 2e-3      # products and result rounded to fp16: 7e-4 and 3e-4
