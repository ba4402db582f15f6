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


@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("rep,G,oc", [(4, 32, 32), (8, 32, 32), (3, 64, 40)])
def test_bfloat16_queries_keep_their_range(rep, G, oc, given):
    """Queries times a power of two give the scores times that power, bit for bit: beyond fp16's largest number (2^16) and
    below its normal ones (2^-14) as well; rows of one call each have their own."""
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(rep)
    n, S = 3, torch.randn(128, 256, generator=g)
    q = torch.randn(1, 2 * rep, 1, 128, generator=g).bfloat16()
    bits, obits = (torch.randint(0, 256, (1, 2, n, G, 32), generator=g, dtype=torch.uint8) for _ in range(2))
    knorm, onorm = (torch.rand(1, 2, n, G, generator=g) + 3).bfloat16(), torch.rand(1, 2, n, G, generator=g).bfloat16()
    idx = torch.stack([torch.randperm(128, generator=g)[:oc] for _ in range(2 * n)]).view(1, 2, n, oc).to(torch.uint8)
    fixed = [t.cuda() for t in (bits, obits, knorm, onorm, idx)]

    def scores(queries):
        qs = (queries.double() @ S.double()).float().cuda() if given else None
        return ops.qjl_gqa_score(*fixed, qs, queries.cuda(), S.cuda()).cpu()

    base = scores(q)
    factor = 2.0 ** torch.tensor([0., 20., -20., 60., -60., 3.]).repeat(2 * rep)[:2 * rep].view(1, -1, 1, 1)
    assert torch.equal(scores((q.float() * factor).bfloat16()), base * factor)
