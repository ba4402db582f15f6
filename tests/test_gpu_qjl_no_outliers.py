"""QJL without outlier channels, through the C entry points (the tensor-level calls refuse the empty index tensor): one block of
32 keys per group and several, sketch and scores, against the CPU oracle."""

import ctypes

import pytest
import torch

from gpu_util import rel_l2
from oracle import qjl as oq

pytestmark = pytest.mark.gpu


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def test_sketch_without_outliers():
    from calibquant_b200._lib import CQ_DTYPE_F16, CQ_DTYPE_F32, lib
    g = torch.Generator().manual_seed(0)
    keys, proj = torch.randn(1, 2, 96, 128, generator=g).half(), torch.randn(256, 128, generator=g)
    groups, idx = keys.reshape(1, 2, 3, 32, 128), torch.empty(1, 2, 3, 0, dtype=torch.uint8)
    ref_kq, ref_koq, _ = oq.qjl_quant(groups, idx, proj, 256)
    k, p, dummy = keys.cuda(), proj.cuda(), torch.zeros(16, dtype=torch.uint8, device="cuda")
    kq, koq = (torch.empty(1, 2, 3, 32, 32, dtype=torch.uint8, device="cuda") for _ in range(2))
    knorm, onorm = (torch.empty(1, 2, 3, 32, dtype=torch.half, device="cuda") for _ in range(2))
    strides = (ctypes.c_int64 * 3)(*k.stride()[:3])
    rc = lib().cq_qjl_build(_ptr(k), 1, 2, 3, 32, 128, strides, _ptr(p), CQ_DTYPE_F32, 256, 256, 0, CQ_DTYPE_F16, _ptr(dummy), _ptr(kq),
                            _ptr(koq), _ptr(knorm), _ptr(onorm), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert (oq.unpack_bits(kq.cpu()) != oq.unpack_bits(ref_kq)).float().mean() < 1e-3
    assert torch.equal(koq.cpu(), ref_koq) and not onorm.any() and not dummy.any()
    assert torch.allclose(knorm.cpu().float(), groups.float().norm(dim=-1), rtol=2.0 ** -10)


@pytest.mark.parametrize("G,rep", [(32, 4), (64, 4), (64, 8), (40, 6)])
def test_scores_without_outliers(G, rep):
    from calibquant_b200._lib import CQ_DTYPE_F16, CQ_DTYPE_F32, lib
    g = torch.Generator().manual_seed(G)
    n, S = 3, torch.randn(128, 256, generator=g)
    q = torch.randn(1, 2 * rep, 1, 128, generator=g).half()
    bits, obits = (torch.randint(0, 256, (1, 2, n, G, 32), generator=g, dtype=torch.uint8) for _ in range(2))
    knorm = torch.rand(1, 2, n, G, generator=g).half() + 1
    onorm, idx = torch.zeros_like(knorm), torch.empty(1, 2, n, 0, dtype=torch.uint8)
    qs = q.float() @ S
    ref = oq.qjl_gqa_score(bits, obits, knorm, onorm, idx, qs, q, S)
    d = [t.cuda() for t in (bits, obits, knorm, onorm, torch.zeros(16, dtype=torch.uint8), qs, q, S)]
    out = torch.empty(1, 2 * rep, n * G, 1, device="cuda")
    rc = lib().cq_qjl_gqa_score(*[_ptr(t) for t in d], CQ_DTYPE_F32, 1, 2, rep, n, G, 128, 256, 256, 0, CQ_DTYPE_F16, _ptr(out), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert rel_l2(out, ref) <= 1e-4
