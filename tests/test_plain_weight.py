"""Which projections the eager decode step may apply without calling their module.  The check of layouts and devices is replaced by
one that lets everything pass, so that the conditions on the module are what decides."""

import types

import pytest
import torch
from torch import nn

from calibquant_b200 import patch_internvl as pi


class _Quantized(torch.Tensor):
    """A weight as weight-only quantization leaves it: a tensor subclass without storage of its own."""

    @staticmethod
    def __new__(cls, shape):
        return torch.Tensor._make_wrapper_subclass(cls, shape, dtype=torch.float32)

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        return NotImplemented if func is not torch.ops.aten.detach.default else args[0]


def _instance_forward(lin):
    lin.forward = types.MethodType(lambda self, x: nn.Linear.forward(self, x) + 1, lin)


def _subclass_weight(lin):
    lin.weight = nn.Parameter(_Quantized((8, 8)), requires_grad=False)


def _pruned_bias(lin):
    lin.bias = nn.Parameter(torch.ones(8))
    from torch.nn.utils import prune
    prune.l1_unstructured(lin, "bias", amount=1)


def _parametrized(lin):
    class Double(nn.Module):
        def forward(self, w):
            return 2 * w
    nn.utils.parametrize.register_parametrization(lin, "weight", Double())


CALLED = {"forward on the instance": _instance_forward, "subclass weight": _subclass_weight, "pruned bias": _pruned_bias,
          "parametrized": _parametrized, "bias": lambda lin: setattr(lin, "bias", nn.Parameter(torch.ones(8))),
          "hook": lambda lin: lin.register_forward_hook(lambda *a: None),
          "pre-hook": lambda lin: lin.register_forward_pre_hook(lambda *a: None)}


@pytest.fixture
def passing(monkeypatch):
    monkeypatch.setattr(pi, "native", lambda: types.SimpleNamespace(small_ok=lambda x, w: True))


@torch.no_grad()
@pytest.mark.parametrize("change", CALLED, ids=str)
def test_module_has_to_be_called(passing, change):
    lin, x = nn.Linear(8, 8, bias=False), torch.zeros(1, 1, 8)
    assert pi._plain_weight(lin, x) is lin.weight
    CALLED[change](lin)
    assert pi._plain_weight(lin, x) is None


@torch.no_grad()
def test_class_forward_replaced(passing, monkeypatch):
    lin, plain = nn.Linear(8, 8, bias=False), nn.Linear.forward
    monkeypatch.setattr(nn.Linear, "forward", lambda self, x: plain(self, x) + 1)
    assert pi._plain_weight(lin, torch.zeros(1, 1, 8)) is None


def test_autograd_and_subclasses_of_linear(passing):
    class Sub(nn.Linear):
        pass
    x = torch.zeros(1, 1, 8)
    assert pi._plain_weight(nn.Linear(8, 8, bias=False), x) is None
    with torch.no_grad():
        assert pi._plain_weight(Sub(8, 8, bias=False), x) is None
