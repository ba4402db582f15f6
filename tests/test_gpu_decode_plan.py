"""Which decode steps run as one launch, and clusters that are larger than their visual span (CTAs with full-precision tokens
alone) or hold more units than their ring, against the CPU oracle."""

import ctypes

import pytest
import torch

from gpu_util import rel_l2
from test_gpu_decode import _run_case

pytestmark = pytest.mark.gpu


def _one_launch(B, hq, hkv, t_vis, t_fp, bits):
    """A step that is one launch needs no scratch but the status word."""
    from calibquant_b200._lib import CQ_DTYPE_BF16, DecodeArgs, lib
    a = DecodeArgs(batch=B, n_q_heads=hq, n_kv_heads=hkv, head_dim=128, t_vis=t_vis, t_fp=t_fp, bits=bits, group_size=32, dtype=CQ_DTYPE_BF16)
    for name in ("q", "out", "k_code", "k_scale", "k_mn", "v_code", "v_scale", "v_mn", "k_fp", "v_fp"):
        setattr(a, name, 4096)      # aligned; nothing is read by the size query
    a.fp_stride_b, a.fp_stride_h = hkv * max(t_fp, 1) * 128, max(t_fp, 1) * 128
    nbytes = lib().cq_decode_attn_workspace_bytes(ctypes.byref(a))
    assert nbytes > 0
    return nbytes == 256


@pytest.mark.parametrize("args,one", [
    ((1, 32, 8, 256, 64, 1), True), ((16, 32, 8, 3328, 232, 1), True), ((4, 32, 8, 5152, 78, 4), True), ((64, 48, 8, 6656, 269, 2), True),
    ((1, 32, 8, 256, 1000, 1), True),       # 37 us in one CTA per KV head, 13.8 apart, 12.6 in clusters of eight
    ((20, 32, 8, 5152, 64, 4), False),      # clusters of one only: 130 us against 80
    ((2, 32, 8, 9216, 0, 4), False),        # half the warps, nine units of a CTA: 21.8 against 16.7
    ((64, 48, 8, 6656, 269, 1), False),     # seven rounds of clusters of four: 183 against 156
    ((80, 32, 8, 3328, 230, 1), False),     # 2.16 rounds: 111 against 107
    ((24, 8, 8, 256, 1000, 1), False),      # eight chunks of a CTA: 45 against 35
    ((8, 32, 8, 32768, 0, 1), False),
])
def test_which_steps_are_one_launch(args, one):
    assert _one_launch(*args) == one


@pytest.mark.parametrize("B,hq,hkv,t_vis,t_txt,bits,dtype,mask", [
    (1, 4, 1, 32, 900, 1, torch.float16, False),         # one group, eight CTAs
    (1, 8, 1, 256, 300, 2, torch.bfloat16, True),        # one unit, clusters of four, eight heads
    (2, 6, 2, 256 + 32, 400, 2, torch.float16, True),    # two ragged units, clusters of four
    (3, 12, 2, 512, 900, 1, torch.bfloat16, False),
    (75, 8, 2, 9 * 256, 0, 1, torch.float16, False),     # nine units of a CTA, eight slots
    (75, 8, 2, 6 * 256, 0, 2, torch.bfloat16, False),    # six units, five slots
    (75, 8, 2, 4 * 256, 0, 4, torch.float16, False),     # four units, three slots
])
def test_uneven_clusters_match_oracle(B, hq, hkv, t_vis, t_txt, bits, dtype, mask):
    from calibquant_b200 import ops
    assert _one_launch(B, hq, hkv, t_vis, t_txt + 41, bits) or t_txt == 0
    out, ref = _run_case(ops, B, hq, hkv, t_vis, t_txt, bits, dtype, seed=t_vis + bits, with_mask=mask)
    assert rel_l2(out, ref) <= (1e-2 if dtype == torch.float16 else 3e-2), rel_l2(out, ref)
    assert ops.device_status() == 0
