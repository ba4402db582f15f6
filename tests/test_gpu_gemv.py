"""The projection of a few rows against an fp32 product: row counts 1-4, lengths that end inside a round of loads, output rows that end
inside a block; and the split + rotation + append that makes the projection itself."""

import pytest
import torch

from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,N,K", [(1, 4096, 4096), (2, 13, 8), (3, 257, 1032), (4, 1000, 6144)])
def test_linear_small(dtype, rows, N, K):
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(N)
    x, w = torch.randn(rows, 1, K, generator=g).to(dtype), (torch.randn(N, K, generator=g) * 0.1).to(dtype)
    out = ops.linear_small(x.cuda(), w.cuda())
    assert out.shape == (rows, 1, N) and out.dtype == dtype
    assert rel_l2(out, x.float() @ w.float().T) <= (5e-4 if dtype == torch.float16 else 4e-3)


def test_rope_split_append_with_weight():
    """The projection made inside the call is the one torch makes: same bits."""
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(3)
    B, Hkv, n_rep, K = 3, 2, 4, 512
    x, w = torch.randn(B, 1, K, generator=g).half().cuda(), (torch.randn(Hkv * (n_rep + 2) * 128, K, generator=g) * 0.1).half().cuda()
    angle = torch.rand(50, 64, generator=g).repeat(1, 2).cuda() * 6
    cos, sin, pos = angle.cos().half(), angle.sin().half(), torch.tensor([[0], [13], [26]], device="cuda")
    c = [torch.zeros(B, Hkv, 9, 128, dtype=torch.half, device="cuda") for _ in range(4)]
    q = ops.rope_split_append(x, cos, sin, pos, Hkv, n_rep, c[0], c[1], append_index=5, weight=w)
    ref = ops.rope_split_append(torch.nn.functional.linear(x, w), cos, sin, pos, Hkv, n_rep, c[2], c[3], append_index=5)
    assert torch.equal(q, ref) and torch.equal(c[0], c[2]) and torch.equal(c[1], c[3])
