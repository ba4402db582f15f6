"""The live token count on the device, advanced by the launch right before the decode step: every step has to see the newest
token.  The keys grow along the query, so that the newest token takes almost all of the probability."""

import pytest
import torch

from test_gpu_calibquant_format import _step_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,t_vis", [(1, 256), (16, 512)])
@pytest.mark.parametrize("fmt", ["uint8", "group"])
def test_step_sees_the_count_of_the_launch_before(fmt, B, t_vis):
    from calibquant_b200 import calibquant as cq, ops
    room, hkv, rep = 96, 2, 4
    q, state, _, _ = _step_inputs(2, B, hkv * rep, hkv, 8, t_vis, 8, torch.float16, seed=B)
    q = q[:, ::rep].repeat_interleave(rep, 1).cuda()      # the heads of a KV head ask the same
    state = {n: t.cuda() for n, t in state.items()}
    g = torch.Generator().manual_seed(1)
    unit = q[:, ::rep].float() / q[:, ::rep].float().norm(dim=-1, keepdim=True) ** 2
    k_fp = (unit * 4 * 128 ** 0.5 * torch.arange(1, room + 1, device="cuda").view(1, 1, room, 1)).half()      # logits 4, 8, 12 ..
    v_fp = torch.randn(B, hkv, room, 128, generator=g).half().cuda()
    if fmt == "group":
        packs = ops.pack_k_per_channel(torch.randn(B, hkv, t_vis, 128, generator=g).half().cuda(), 32, 2), \
            ops.pack_v_per_token(torch.randn(B, hkv, t_vis, 128, generator=g).half().cuda(), 32, 2)
    live = torch.full((1,), 16, dtype=torch.int32, device="cuda")
    outs = []
    for _ in range(room - 16):
        live.add_(1)
        if fmt == "group":
            outs.append(ops.decode_attention(q, *packs, k_fp, v_fp, 8, 2, t_fp_dev=live))
        else:
            outs.append(cq.decode_attention(q, state, k_fp, v_fp, 2, 8, t_fp_dev=live))
    for i, out in enumerate(outs):      # e^-4 of the probability is left to the others
        newest = v_fp[:, :, 16 + i].repeat_interleave(rep, 1).float()
        assert (out[:, :, 0].float() - newest).norm() <= 0.1 * newest.norm()


def test_uint8_step_takes_an_int64_count():
    from calibquant_b200 import calibquant as cq
    q, state, k_fp, v_fp = _step_inputs(2, 1, 8, 2, 8, 64, 24, torch.float16, seed=4)
    args = q.cuda(), {n: t.cuda() for n, t in state.items()}, k_fp.cuda(), v_fp.cuda(), 2, 8
    want, got = (cq.decode_attention(*args, t_fp_dev=torch.tensor([20], dtype=t, device="cuda")) for t in (torch.int32, torch.int64))
    assert torch.equal(got, want)
