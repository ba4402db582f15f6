"""What the eager decode step of the patched forward refuses and accepts: positions as torch indexes the rotary table with them,
projections that have to be called."""

import os
import types

import pytest
import torch

from test_gpu_forward import _layer

pytestmark = pytest.mark.gpu

T_VIS, B = 256, 2
T = 41 + T_VIS + 7


@pytest.fixture
def layer(monkeypatch):
    from calibquant_b200 import patch_internvl as pi
    shell = _layer(8, 2, seed=1)
    pi.patch_model(shell, "calibquant")
    monkeypatch.setattr(pi, "BITS_KV", 2)
    monkeypatch.setattr(pi, "SCALE_K", 1)
    monkeypatch.setattr(pi, "SCALE_V", 1)
    monkeypatch.setitem(os.environ, "IMAGE_TOKEN_NUM", str(T_VIS))
    return shell.cuda().language_model.model.layers[0].attention


def _prompt(attn):
    g = torch.Generator().manual_seed(5)
    h = (torch.randn(B, T + 1, 1024, generator=g) * 0.5).half().cuda()
    pos = torch.arange(T, device="cuda").unsqueeze(0).expand(B, T)
    _, _, past = attn(h[:, :T], position_ids=pos, use_cache=True)
    return h[:, T:], past


@torch.no_grad()
def _step(attn, position, **kw):
    x, past = _prompt(attn)
    out, _, past = attn(x, position_ids=torch.tensor(position, device="cuda").view(-1, 1), past_key_value=kw.get("past", past), use_cache=True)
    return out, past


def test_positions_index_the_table_as_torch_does(layer):
    """The table of a step has a row per token so far (T + 1 rows): negative positions count from its end, others outside it
    are refused - the rows come out as not-a-number, the status says so, and the next step on the stream raises once."""
    from calibquant_b200 import _lib, ops
    want, _ = _step(layer, [T, T - 3])
    got, _ = _step(layer, [-1, T - 3])
    assert torch.equal(got, want)
    for bad in (T + 1, -T - 2, 1 << 40):
        out, past = _step(layer, [T, bad])
        assert torch.equal(out[0], want[0]) and torch.isnan(out[1].float()).all()
        assert torch.isnan(past[0][1, :, -1].float()).all()      # the key appended
        assert ops.device_status() == _lib.CQ_ERR_BAD_ARG
        with pytest.raises(RuntimeError, match="position_ids"):
            _step(layer, [T, T])
        assert ops.device_status() == 0
        assert torch.equal(_step(layer, [T, T - 3])[0], want)


def test_step_without_the_past_has_a_table_of_one_row(layer):
    out, _ = _step(layer, [T, T], past=None)
    assert torch.isnan(out.float()).all()
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="position_ids"):
        _step(layer, [T, T])


def test_direct_calls_clamp_as_documented():
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(2)
    qkv, table = torch.randn(1, 1, 6 * 128, generator=g).half().cuda(), torch.randn(2, 9, 128, generator=g).half().cuda()
    outs = []
    for pos in (8, 99):
        cache = torch.zeros(2, 1, 1, 4, 128, dtype=torch.half, device="cuda")
        outs.append(ops.rope_split_append(qkv, *table, torch.tensor([[pos]], device="cuda"), 1, 4, *cache, append_index=0))
    assert torch.equal(*outs) and ops.device_status() == 0


@pytest.mark.parametrize("name", ["wqkv", "wo"])
def test_wrapped_projection_is_called(layer, name):
    want, _ = _step(layer, [T, T])
    lin, calls = getattr(layer, name), []

    def wrapped(self, x):
        calls.append(x.shape[1])
        return torch.nn.functional.linear(x, self.weight)

    lin.forward = types.MethodType(wrapped, lin)
    out, _ = _step(layer, [T, T])
    assert calls == [T, 1]
    assert (out.float() - want.float()).norm() <= 1e-2 * want.float().norm()


@pytest.mark.parametrize("dtype,device", [(torch.int32, "cuda"), (torch.int64, "cpu"), (torch.int32, "cpu")])
def test_positions_of_other_types_and_on_the_host(layer, dtype, device):
    want, _ = _step(layer, [T, T - 3])
    with torch.no_grad():
        x, past = _prompt(layer)
        pos = torch.tensor([[T], [T - 3]], dtype=dtype, device=device)
        out, _, _ = layer(x, position_ids=pos, past_key_value=past, use_cache=True)
    assert torch.equal(out, want)


@torch.no_grad()
def test_more_rows_than_the_cache_holds(layer):
    x, past = _prompt(layer)
    length = layer._text_cache.length
    with pytest.raises(ValueError, match="does not hold"):
        layer(torch.cat([x, x]), position_ids=torch.full((2 * B, 1), T, device="cuda"), past_key_value=past, use_cache=True)
    assert layer._text_cache.length == length


def test_append_to_a_smaller_cache():
    from calibquant_b200 import ops
    qkv, table = torch.zeros(2, 1, 12 * 128, device="cuda").half(), torch.zeros(2, 9, 128, device="cuda").half()
    pos = torch.zeros(2, 1, dtype=torch.int64, device="cuda")
    for shape in ((1, 2, 4, 128), (2, 1, 4, 128)):
        cache = torch.zeros(2, *shape, device="cuda").half()
        with pytest.raises(ValueError, match="does not hold"):
            ops.rope_split_append(qkv, *table, pos, 2, 4, *cache, append_index=0)
