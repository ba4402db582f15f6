"""The QJL sketch quantizer at group sizes and sketch sizes other than (32, 256): against the CPU oracle, and on the tensor
cores rather than the CUDA cores."""

import ctypes

import pytest
import torch

from oracle import qjl as oq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,G,sketch,o_sketch,oc", [(1, 1, 32, 32, 4), (3, 31, 128, 128, 32), (5, 33, 256, 64, 8),
                                                    (4, 64, 256, 256, 32), (3, 100, 224, 96, 128), (300, 32, 128, 128, 32)])
def test_other_sizes_match_oracle(dtype, n, G, sketch, o_sketch, oc):
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(G + sketch)
    keys = (torch.randn(1, 1, n, G, 128, generator=g) * torch.exp(0.5 * torch.randn(128, generator=g))).to(dtype)
    idx = torch.stack([torch.randperm(128, generator=g)[:oc] for _ in range(n)]).view(1, 1, n, oc).to(torch.uint8)
    proj = torch.randn(sketch, 128, generator=g)
    kq, koq, norms = (t.cpu() for t in ops.qjl_quant(keys.cuda(), idx.cuda(), proj.cuda(), o_sketch))
    r_kq, r_koq, r_norms = oq.qjl_quant(keys, idx, proj, o_sketch)
    s_in, s_out = oq.sketches(keys, idx, proj)
    for got, ref, val in ((kq, r_kq, s_in), (koq, r_koq, s_out[..., :o_sketch])):
        diff = oq.unpack_bits(got) != oq.unpack_bits(ref)
        assert (val[diff].abs() < 1e-3 * val.abs().mean()).all()      # sums at rounding distance of zero
    ulp = 2.0 ** (-10 if dtype == torch.float16 else -7)
    assert (norms.float() - r_norms.float()).abs().le(r_norms.float() * ulp + 1e-6).all()


@pytest.mark.parametrize("G,sketch", [(64, 256), (32, 128)])
def test_other_sizes_run_on_the_tensor_cores(G, sketch):
    """Keys that start off a 16-byte boundary are left to the CUDA cores; aligned ones have to be clearly faster (about four
    times at 256 projections)."""
    from calibquant_b200._lib import CQ_DTYPE_F16, CQ_DTYPE_F32, lib
    tokens = 8 * 16384
    buf = torch.randn(tokens * 128 + 8, device="cuda").half()
    idx = torch.arange(32, dtype=torch.uint8, device="cuda").repeat(tokens // G)
    proj = torch.randn(sketch, 128, device="cuda")
    kq, koq = (torch.empty(tokens, sketch // 8, dtype=torch.uint8, device="cuda") for _ in range(2))
    norms = torch.empty(tokens, dtype=torch.half, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def ms(offset):
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
        for e in ev:
            e.record()
            rc = lib().cq_qjl_quant(p(buf[offset:]), p(idx), p(proj), CQ_DTYPE_F32, tokens // G, G, 128, sketch, sketch, 32, CQ_DTYPE_F16,
                                    p(kq), p(koq), p(norms), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == 0
        torch.cuda.synchronize()
        return min(ev[i].elapsed_time(ev[i + 1]) for i in range(3))

    assert 1.5 * ms(0) < ms(4)
