"""Roundings of the logit calibration in the single-launch decode step on the uint8 format: fp16 rows without a mask round
product and sum once, rows with a mask every operation, as torch does."""

import pytest
import torch

from gpu_util import rel_l2
from oracle import calibquant_format as cqf
from test_gpu_calibquant_format import _step_inputs

pytestmark = pytest.mark.gpu


def _calibrate_rounding_once(s):
    hi, lo = s.amax(dim=(2, 3), keepdim=True), s.amin(dim=(2, 3), keepdim=True)
    n = (s - lo) / (hi - lo + 1e-8)
    return (n.double() * (hi + (-3) - lo).double() + lo.double()).to(s.dtype)


@pytest.mark.parametrize("masked", [False, True])
def test_fp16_calibration_roundings(monkeypatch, masked):
    from calibquant_b200 import calibquant as cq
    q, state, k_fp, v_fp = _step_inputs(1, 4, 16, 4, 41, 1024, 30, torch.float16, seed=3)
    mask = torch.zeros(4, 1024 + 71, dtype=torch.float16, device="cuda") if masked else None
    out = cq.decode_attention(q.cuda(), {n: t.cuda() for n, t in state.items()}, k_fp.cuda(), v_fp.cuda(), 1, 41, mask=mask)
    two = cqf.decode_attention(q, state, k_fp, v_fp, 1, 41)
    monkeypatch.setattr(cqf, "calibrate", _calibrate_rounding_once)
    one = cqf.decode_attention(q, state, k_fp, v_fp, 1, 41)
    # the order of fp32 sums is all that is left between the kernel and the form it follows
    near, far = (two, one) if masked else (one, two)
    assert rel_l2(out, near) < 0.5 * rel_l2(out, far)
