"""The one-launch sketch of strided keys (tcgen05) against the torch ops and the CPU-oracle quantizer it stands for: tiles
of four groups that end inside a (batch, head) run, a single group, outlier counts from eight to all channels, short outlier
sketches, both data types and projections of either type."""

import pytest
import torch

from oracle import qjl as oq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,H,T,oc,o_sketch,same", [(1, 1, 32, 32, 256, False), (2, 3, 160, 32, 256, False), (1, 2, 1216, 8, 128, True),
                                                    (3, 8, 1312, 128, 32, False)])
def test_build_matches_torch_and_oracle(dtype, B, H, T, oc, o_sketch, same):
    from calibquant_b200 import ops
    from calibquant_b200._lib import lib
    g = torch.Generator().manual_seed(T + oc)
    full = (torch.randn(B, H, T + 9, 128, generator=g) * torch.exp(0.7 * torch.randn(128, generator=g))).to(dtype)
    proj = torch.randn(256, 128, generator=g)
    proj = proj.to(dtype) if same else proj
    idx, kq, koq, onorm, knorm = (t.cpu() for t in ops.qjl_build(full.cuda()[:, :, :T], proj.cuda(), o_sketch, oc))
    groups = full[:, :, :T].reshape(B, H, T // 32, 32, 128)
    norms = groups.float().square().sum(-2).sqrt().to(dtype)
    # the chosen channels are the oc largest (up to one rounding step of the data type), largest first
    picked = torch.gather(norms.float(), -1, idx.long())
    best = norms.float().sort(dim=-1, descending=True).values[..., :oc]
    assert torch.allclose(picked, best, rtol=2e-3 if dtype == torch.float16 else 1.6e-2, atol=0)
    assert all(len(set(r.tolist())) == oc for r in idx.reshape(-1, oc))
    ref_kq, ref_koq, ref_onorm = oq.qjl_quant(groups, idx, proj, o_sketch)
    for mine, ref in ((kq, ref_kq), (koq, ref_koq)):
        diff = (mine ^ ref).to(torch.int32)
        flipped = sum(int(((diff >> i) & 1).sum()) for i in range(8))
        assert flipped <= 1e-4 * 8 * diff.numel(), flipped
    tol = 2e-3 if dtype == torch.float16 else 1.6e-2
    assert torch.allclose(onorm.float(), ref_onorm.float(), rtol=tol, atol=1e-6)
    assert torch.allclose(knorm.float(), groups.float().norm(dim=-1), rtol=tol, atol=1e-6)
    assert lib().cq_qjl_status() == 0
