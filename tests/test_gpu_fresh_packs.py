"""A decode step directly behind the launch that wrote its packed operands, whichever of them that was (keys, values, a copy made
contiguous on the way in): the result is the one of the same operands at rest."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", ["keys", "values", "copy"])
@pytest.mark.parametrize("B,t_vis,bits", [(1, 256, 1), (2, 800, 2), (4, 3328, 4), (2, 32768, 1), (1, 33024, 4)])
def test_step_behind_the_pack(B, t_vis, bits, last):
    from calibquant_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(t_vis)
    q = torch.randn(B, 32, 1, 128, generator=g, device="cuda").half()
    fp = torch.randn(2, B, 8, 64, 128, generator=g, device="cuda").half()
    for _ in range(6):
        k, v = (torch.randn(B, 8, t_vis, 128, generator=g, device="cuda").half() for _ in range(2))
        torch.cuda.synchronize()
        if last == "keys":
            vp = ops.pack_v_per_token(v, 32, bits)
            kp = ops.pack_k_per_channel(k, 32, bits)
        else:
            kp = ops.pack_k_per_channel(k, 32, bits)
            vp = ops.pack_v_per_token(v, 32, bits)
        if last == "copy":      # strided views: the step itself has to copy them
            kp, vp = ([torch.stack([t, t], dim=-1)[..., 0] for t in p] for p in (kp, vp))
            torch.cuda.synchronize()
        out = ops.decode_attention(q, kp, vp, *fp, 41, bits)
        torch.cuda.synchronize()
        assert torch.equal(out, ops.decode_attention(q, [t.contiguous() for t in kp], [t.contiguous() for t in vp], *fp, 41, bits))
