"""Precision of the QJL score estimate's sums, against 64-bit arithmetic."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _one_group(q, S, signs=255):
    """Scores of one group of 32 keys of unit norm without an outlier part; channels 0-31 are the outlier channels."""
    from calibquant_b200.qjl import qjl_kernel
    rep, sketch = q.shape[1], S.shape[1]
    idx = torch.arange(32, dtype=torch.uint8).view(1, 1, 1, 32)
    bits = torch.full((1, 1, 1, 32, sketch // 8), signs, dtype=torch.uint8)
    norm = torch.ones(1, 1, 1, 32, dtype=q.dtype)
    qs = (q.double() @ S.double()).float()
    args = (bits, bits, norm, torch.zeros_like(norm), idx, qs, q, S)
    return qjl_kernel.qjl_gqa_score(*[t.cuda() for t in args]).cpu().double().view(rep, 32)


@pytest.mark.parametrize("rep", [1, 4, 5, 8])
def test_sums_of_one_sign(rep):
    """All signs and terms positive, over twelve binary orders: every truncated addition counts. The final rounding, the
    rounding of q S and of the remainders leave about one unit of 2^-23; sixteen truncations in a row were eight."""
    for seed in range(4):
        g = torch.Generator().manual_seed(seed)
        S = torch.exp2(-12 * torch.rand(128, 256, generator=g)).half().float()
        q = torch.zeros(1, rep, 1, 128, dtype=torch.float16)
        q[..., 64:] = 1.0
        exact = math.sqrt(math.pi / 2) / 256 * (q[0, :, 0].double() @ S.double()).sum(-1, keepdim=True)
        assert ((_one_group(q, S) - exact) / exact).abs().max() <= 3 * 2.0 ** -23
