"""``ops.linear_small`` on both sides of the row length from which it is a matrix product, against fp32."""

import pytest
import torch

from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [4096, 4104, 6144])
@pytest.mark.parametrize("shape", [(1, 1), (2, 1), (4, 1), (3,)])
def test_row_lengths(K, shape):
    from calibquant_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = torch.randn(*shape, K, generator=g, device="cuda").bfloat16(), torch.randn(264, K, generator=g, device="cuda").bfloat16()
    out = ops.linear_small(x, w)
    assert out.shape == (*shape, 264) and out.dtype == x.dtype
    assert rel_l2(out, x.float() @ w.float().t()) <= 2.0 ** -8


@pytest.mark.parametrize("K", [4096, 6144])
def test_more_rows_are_refused(K):
    from calibquant_b200 import ops
    with pytest.raises(ValueError):
        ops.linear_small(torch.zeros(5, K, device="cuda").half(), torch.zeros(16, K, device="cuda").half())
