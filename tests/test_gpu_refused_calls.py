"""Tensor-level calls that the Python checks refused before the entry points were moved into the extension module, and that it has
to refuse as well."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _half(*shape):
    return torch.randn(*shape, device="cuda").half()


def _packs(B=1, T=64):
    from calibquant_b200 import ops
    return ops.pack_k_per_channel(_half(B, 2, T, 128), 32, 2), ops.pack_v_per_token(_half(B, 2, T, 128), 32, 2)


def _u8(B=1, T=64):
    from calibquant_b200 import calibquant as cq
    (ek, sk, zk), (ev, sv, zv) = (cq.quant_encode(_half(B, T, 2, 128), 2) for _ in range(2))
    return {"enc_k": ek, "enc_v": ev, "scale_key": sk, "zero_point_key": zk, "scale_value": sv, "zero_point_value": zv}


def test_several_query_rows():
    from calibquant_b200 import calibquant as cq, ops
    fp = _half(1, 2, 8, 128)
    with pytest.raises(RuntimeError):
        ops.decode_attention(_half(1, 8, 2, 128), *_packs(), fp, fp, 4, 2)
    with pytest.raises(RuntimeError):
        cq.decode_attention(_half(1, 8, 2, 128), _u8(), fp, fp, 2, 4)
    with pytest.raises(ValueError):
        cq.decode_attention(_half(1, 8, 128), _u8(), fp, fp, 2, 4)


def test_other_numbers_of_dimensions():
    from calibquant_b200 import calibquant as cq, ops
    with pytest.raises(ValueError):
        cq.quant_encode(_half(1, 64, 2, 128, 2), 2)
    with pytest.raises(ValueError):
        ops.prefill_attention(_half(1, 64, 8, 128, 2), _half(1, 64, 2, 128), _half(1, 64, 2, 128))
    idx, proj = torch.zeros(1, 2, 2, 8, dtype=torch.uint8, device="cuda"), torch.randn(256, 128, device="cuda")
    with pytest.raises(ValueError):
        ops.qjl_quant(_half(1, 2, 2, 32, 128, 2), idx, proj, 256)
    bits, norm = torch.zeros(1, 2, 2, 32, 32, 2, dtype=torch.uint8, device="cuda"), _half(1, 2, 2, 32)
    with pytest.raises(ValueError):
        ops.qjl_gqa_score(bits, bits, norm, norm, idx, None, _half(1, 8, 1, 128), proj.t().contiguous())


def test_sizes_of_zero_raise():
    """What Python refused as a division by zero must not end the process."""
    from calibquant_b200 import calibquant as cq, ops
    from calibquant_b200._lib import native
    kp, vp = _packs()
    fp, idx = _half(0, 2, 8, 128), torch.zeros(1, 0, 2, 8, dtype=torch.uint8, device="cuda")
    bits, norm = torch.zeros(1, 0, 2, 32, 32, dtype=torch.uint8, device="cuda"), _half(1, 0, 2, 32)
    calls = [lambda: ops.pack_v_per_token(_half(1, 2, 64, 128), 0, 2), lambda: ops.pack_k_per_channel(_half(1, 2, 64, 128), 0, 2),
             lambda: ops.pack_last_dim(_half(1, 2, 64, 128), 0, 2), lambda: native().pack_last_dim(_half(1, 2, 64, 128), 0, 2),
             lambda: ops.qbmm(32, _half(1, 8, 1, 64), *vp, 0), lambda: cq.decode_attention(_half(0, 8, 1, 128), _u8(), fp, fp, 2, 4),
             lambda: ops.qjl_gqa_score(bits, bits, norm, norm, idx, None, _half(1, 8, 1, 128), torch.randn(128, 256, device="cuda"))]
    for call in calls:
        with pytest.raises(ZeroDivisionError):
            call()
