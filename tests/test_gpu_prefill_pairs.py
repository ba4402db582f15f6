"""Prefill attention at the edges of its work items: an odd and an even number of query heads per KV head (adjacent query
tiles / the same queries of two heads share an item), prompts that end on, just behind and just before a tile, and grids
whose CTAs take over several items of different lengths.  And the split + rotation at token counts around the point where a
token's heads are spread over several warps."""

import pytest
import torch

from oracle import prefill as oracle_prefill
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rep,T,B,Hkv", [(1, 129, 2, 3), (3, 257, 1, 2), (1, 640, 4, 16), (2, 128, 1, 2), (2, 129, 1, 2), (4, 256, 3, 8),
                                           (2, 384, 5, 32), (6, 511, 2, 4)])
def test_items(n_rep, T, B, Hkv):
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(T + n_rep)
    q = torch.randn(B, T, Hkv * n_rep, 128, generator=g).half()
    k, v = (torch.randn(B, T, Hkv, 128, generator=g).half() for _ in range(2))
    ref = oracle_prefill.causal_attention(q, k, v)
    out = ops.prefill_attention(q.cuda(), k.cuda(), v.cuda())
    assert rel_l2(out, ref) <= 5e-3
    worst = (out.cpu().float() - ref.float()).abs().amax(dim=(1, 3))      # per (batch, head): a tile in the wrong place shows
    assert float(worst.max()) <= 2e-2


@pytest.mark.parametrize("B,T,Hkv,n_rep", [(1, 1, 8, 4), (1, 300, 3, 5), (2, 147, 8, 1), (2, 1184, 8, 6)])
def test_rope_split_parts(B, T, Hkv, n_rep):
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(T)
    qkv = torch.randn(B, T, Hkv, n_rep + 2, 128, generator=g).half().cuda()
    angle = torch.rand(T + 3, 64, generator=g).repeat(1, 2).cuda()
    cos, sin = angle.cos().half(), angle.sin().half()
    vis_start = min(5, T - 1)
    n_vis = (T - vis_start) // 2
    kc = torch.zeros(B, Hkv, T - n_vis + 4, 128, dtype=torch.half, device="cuda")
    vc = torch.zeros_like(kc)
    q, k, v = ops.prefill_rope_split(qkv.view(B, T, -1), cos, sin, None, Hkv, n_rep, kc, vc, vis_start, n_vis)
    x = qkv[:, :, :, : n_rep + 1]
    rot = torch.cat((-x[..., 64:], x[..., :64]), dim=-1)
    c, s = cos[:T, None, None], sin[:T, None, None]
    ref = torch.addcmul(x * c, rot, s)
    assert torch.equal(q, ref[:, :, :, :n_rep].reshape(B, T, -1, 128))
    assert torch.equal(k, ref[:, :, :, n_rep])
    keep = [t for t in range(T) if not vis_start <= t < vis_start + n_vis]
    assert torch.equal(kc[:, :, : len(keep)], k[:, keep].transpose(1, 2))
    assert torch.equal(vc[:, :, : len(keep)], qkv[:, keep, :, -1].transpose(1, 2))
