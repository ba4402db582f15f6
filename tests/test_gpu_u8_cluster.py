"""The single-launch decode step on the uint8 format at the edges of its split (items of 64 visual tokens, tiles of 16
full-precision tokens, clusters of 1 to 8), against the CPU oracle."""

import pytest
import torch

from gpu_util import rel_l2
from oracle import calibquant_format as cqf
from test_gpu_calibquant_format import _step_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 2, 4])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,hq,hkv,t_vis,t_txt,sys_len", [
    (1, 1, 1, 1, 0, 1),          # one key of each kind
    (1, 6, 1, 63, 5, 41),        # less than an item, six heads
    (2, 8, 2, 65, 90, 3),        # one key past an item, a system span that ends inside a tile of 16
    (1, 16, 2, 1999, 210, 41),   # odd span over eight CTAs, eight heads
    (40, 8, 2, 333, 17, 41),     # clusters of two
    (80, 8, 2, 100, 4, 0),       # no system tokens, one CTA per KV head
])
def test_u8_single_launch_edges(bits, dtype, B, hq, hkv, t_vis, t_txt, sys_len):
    from calibquant_b200 import calibquant as cq, ops
    q, state, k_fp, v_fp = _step_inputs(bits, B, hq, hkv, sys_len, t_vis, t_txt, dtype, seed=t_vis + bits)
    ref = cqf.decode_attention(q, state, k_fp, v_fp, bits, sys_len)
    out = cq.decode_attention(q.cuda(), {n: t.cuda() for n, t in state.items()}, k_fp.cuda(), v_fp.cuda(), bits, sys_len)
    # a span of a single key has scale 0 and an infinite zero point in every implementation: compare where finite
    ok = torch.isfinite(ref.float()) & torch.isfinite(out.cpu().float())
    assert torch.equal(torch.isfinite(ref.float()), torch.isfinite(out.cpu().float()))
    assert rel_l2(torch.where(ok, out.cpu().float(), 0.), torch.where(ok, ref.float(), 0.)) <= 1e-2
    assert ops.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("q_scale,fp_scale", [(0.02, 1.0), (1.0, 4.0), (1.0, 0.05)])
def test_u8_maximum_from_the_extremes(dtype, q_scale, fp_scale):
    """Scores within 3 of each other, which the calibration turns around; full-precision scores of some CTAs far above the visual
    ones, so that a CTA's maximum is not the cluster's; far below.  bfloat16 probabilities (2^-9) set the bar."""
    from calibquant_b200 import calibquant as cq, ops
    q, state, k_fp, v_fp = _step_inputs(1, 2, 8, 2, 5, 1111, 60, dtype, seed=7)
    q, k_fp = q * q_scale, k_fp * fp_scale
    ref = cqf.decode_attention(q, state, k_fp, v_fp, 1, 5)
    out = cq.decode_attention(q.cuda(), {n: t.cuda() for n, t in state.items()}, k_fp.cuda(), v_fp.cuda(), 1, 5)
    assert rel_l2(out.cpu(), ref) <= 1e-2
    assert ops.device_status() == 0
