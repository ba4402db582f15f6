"""The single-launch decode step (one cluster per KV head) at the edges of its tiling, against the CPU oracle: one group,
one unit, more units than ring slots, units that do not divide over the cluster, ragged spans with an odd number of
groups, more full-precision tokens than one block of 128 per CTA, every head grouping."""

import pytest
import torch

from gpu_util import rel_l2
from test_gpu_decode import _run_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from calibquant_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("bits", [1, 2, 4])
@pytest.mark.parametrize("B,hq,hkv,t_vis,t_txt,dtype,mask", [
    (1, 1, 1, 32, 0, torch.float16, False),            # one group, one head, one CTA
    (1, 4, 1, 256, 300, torch.float16, True),          # one unit; 341 full-precision tokens on one CTA
    (2, 8, 2, 2304, 3, torch.bfloat16, False),         # nine units over eight CTAs
    (1, 12, 2, 8 * 2560, 150, torch.float16, False),   # ten units per CTA: more than the ring holds, six heads
    (18, 16, 2, 1056, 20, torch.float16, False),       # 33 groups over clusters of four, eight heads
    (40, 8, 2, 768, 9, torch.bfloat16, True),          # clusters of two
    (3, 5, 1, 1600 + 32, 70, torch.float16, True),     # odd number of groups, five heads
])
def test_single_launch_step_edges(ops, bits, B, hq, hkv, t_vis, t_txt, dtype, mask):
    out, ref = _run_case(ops, B, hq, hkv, t_vis, t_txt, bits, dtype, seed=bits + t_vis + hq, with_mask=mask)
    assert rel_l2(out, ref) <= (1e-2 if dtype == torch.float16 else 3e-2), rel_l2(out, ref)
    assert ops.device_status() == 0


@pytest.mark.parametrize("B,hq,hkv,t_vis,t_txt,bits,dtype", [
    (34, 16, 8, 4 * 256, 5, 1, torch.float16),         # one CTA per pair would leave the second round nearly empty: separate launches
    (70, 32, 8, 2 * 256, 3, 2, torch.bfloat16),        # two rounds of one CTA per pair, the last one not full
    (100, 6, 3, 256 + 96, 0, 1, torch.float16),        # just above one round, ragged span
    (24, 64, 8, 24 * 256, 0, 1, torch.float16),        # eight heads: rounds of clusters of two
])
def test_more_pairs_than_resident_clusters(ops, B, hq, hkv, t_vis, t_txt, bits, dtype):
    out, ref = _run_case(ops, B, hq, hkv, t_vis, t_txt, bits, dtype, seed=bits + t_vis + hq)
    assert rel_l2(out, ref) <= (1e-2 if dtype == torch.float16 else 3e-2), rel_l2(out, ref)
    assert ops.device_status() == 0
