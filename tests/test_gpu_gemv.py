"""The projections of a few rows: against an fp32 product, and the fused projection + split + rotation + append against the two
steps it stands for; row counts 1-4, lengths that end inside a round of loads, output rows that end inside a block."""

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


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,Hkv,n_rep,K", [(1, 8, 4, 4096), (2, 1, 1, 136), (3, 3, 6, 512), (4, 2, 2, 1024)])
def test_qkv_rope_append(dtype, B, Hkv, n_rep, K):
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(K)
    x = torch.randn(B, 1, K, generator=g).to(dtype).cuda()
    w = (torch.randn(Hkv * (n_rep + 2) * 128, K, generator=g) * 0.1).to(dtype).cuda()
    angle = torch.rand(50, 64, generator=g).repeat(1, 2).cuda() * 6
    cos, sin = angle.cos().to(dtype), angle.sin().to(dtype)
    pos = torch.tensor([[i * 13] for i in range(B)], device="cuda")
    caches = [torch.zeros(B, Hkv, 9, 128, dtype=dtype, device="cuda") for _ in range(4)]
    q = ops.qkv_rope_append(x, w, cos, sin, pos, Hkv, n_rep, caches[0], caches[1], 5)
    ref_q = ops.rope_split_append((x.float() @ w.float().T).to(dtype), cos, sin, pos, Hkv, n_rep, caches[2], caches[3], append_index=5)
    tol = 1e-3 if dtype == torch.float16 else 8e-3      # sums in another order, rounded to the data type
    for mine, ref in ((q, ref_q), (caches[0], caches[2]), (caches[1], caches[3])):
        assert rel_l2(mine, ref.cpu()) <= tol
    assert int((caches[0] != 0).any(-1).sum()) == B * Hkv      # one token row per head and request
