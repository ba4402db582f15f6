"""QJL score estimate on the 5th-generation tensor cores, against 64-bit arithmetic of the oracle's formula: calls of one unit (4
groups) a CTA with every form of the operands, and calls of several tiles (4 to 16 groups) a CTA."""

import math

import pytest
import torch

from gpu_util import rel_l2
from oracle import qjl as oq

pytestmark = pytest.mark.gpu


def _exact(bits, obits, knorm, onorm, idx, qs, q, S):
    """The oracle's formula in 64 bits; a channel named more than once counts as often."""
    hkv, n, s, so = bits.shape[1], bits.shape[2], bits.shape[-1] * 8, obits.shape[-1] * 8
    qd, m = q.double().view(q.shape[0], hkv, -1, 128), torch.zeros(*idx.shape[:3], 128, dtype=torch.float64)
    m.scatter_add_(-1, idx.long(), torch.ones(idx.shape, dtype=torch.float64))
    q_out = torch.einsum("bhrd,bhnd,ds->bhnrs", qd, m, S.double())
    q_in = (qs.double().view(*qd.shape[:3], s) if qs is not None else qd @ S.double()).unsqueeze(2) - q_out
    sgn, sgn_o = oq.unpack_bits(bits).double() * 2 - 1, oq.unpack_bits(obits).double() * 2 - 1
    no = onorm.double().unsqueeze(2)
    ni = (knorm.double().unsqueeze(2).pow(2) - no.pow(2)).clamp_min(0).sqrt()
    score = ni / s * torch.einsum("bhngs,bhnrs->bhrng", sgn, q_in) + no / so * torch.einsum("bhngs,bhnrs->bhrng", sgn_o, q_out[..., :so])
    return (math.sqrt(math.pi / 2) * score).reshape(q.shape[0], q.shape[1], n * 32, 1)


@pytest.mark.parametrize("n,rep,oc,so,given", [(1, 1, 32, 256, False), (3, 2, 8, 128, True), (4, 3, 32, 256, True), (17, 4, 32, 256, False),
                                               (33, 4, 40, 128, False), (70, 4, 1, 256, False), (16, 4, 128, 256, False)])
@pytest.mark.parametrize("dtype,pdtype", [(torch.half, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_against_64_bits(n, rep, oc, so, given, dtype, pdtype):
    """The projection is carried to 2^-22, sums are truncated sixteen times at 2^-23 or so: 1e-5 in all (measured: 1e-6)."""
    from calibquant_b200 import ops
    from calibquant_b200._lib import lib
    g = torch.Generator().manual_seed(100 * n + rep)
    S = torch.randn(128, 256, generator=g).to(pdtype)
    q = (torch.randn(3, 2 * rep, 1, 128, generator=g) * 3).to(dtype)
    bits, obits = (torch.randint(0, 256, (3, 2, n, 32, w // 8), generator=g, dtype=torch.uint8) for w in (256, so))
    onorm = (torch.rand(3, 2, n, 32, generator=g) * 4).to(dtype)
    knorm = (onorm.float() + torch.rand(3, 2, n, 32, generator=g) * 6).to(dtype)
    idx = torch.stack([torch.randperm(128, generator=g)[:oc] for _ in range(6 * n)]).view(3, 2, n, oc).to(torch.uint8)
    if oc > 1:
        idx[:, 1, 0, 1] = idx[:, 1, 0, 0]      # named twice: exact in fp16
    qs = (q.float() @ S.float()) if given else None
    ref = _exact(bits, obits, knorm, onorm, idx, qs, q, S)
    dev = [None if t is None else t.cuda() for t in (bits, obits, knorm, onorm, idx, qs, q, S)]
    got = ops.qjl_gqa_score(*dev).cpu()
    assert rel_l2(got, ref) <= 1e-5
    for head in range(2 * rep):
        assert rel_l2(got[:, head], ref[:, head]) <= 2e-5
    assert lib().cq_qjl_status() == 0


@pytest.mark.parametrize("kbh,n,rep,so,given", [
    (64, 70, 4, 256, False),       # a ragged last tile
    (64, 40, 3, 128, True),
    (40, 99, 4, 256, False),       # heads change within a CTA
    (160, 18, 4, 256, True),
    (16, 257, 1, 128, False),
    (37, 131, 2, 256, False),
    (1200, 4, 4, 256, False),      # a head a unit: more tiles a CTA than the ring of totals has slots
    (1300, 3, 3, 128, True),
])
def test_many_tiles_a_cta(kbh, n, rep, so, given):
    """Every barrier in its later phases, both operand buffers, the ring of totals, changes of the head within a CTA.  More than four
    units a CTA make at least two tiles, whatever their size (four units at most).  Another query for every head; bounds as
    above."""
    from calibquant_b200 import ops
    from calibquant_b200._lib import lib
    assert kbh * -(-n // 4) > 4 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(kbh)
    rand = lambda *shape: torch.rand(*shape, generator=g, device="cuda")
    S = torch.randn(128, 256, generator=g, device="cuda")
    q = (torch.randn(1, kbh * rep, 1, 128, generator=g, device="cuda") * (1 + 5 * rand(1, kbh * rep, 1, 1))).half()
    bits, obits = (torch.randint(0, 256, (1, kbh, n, 32, w // 8), generator=g, dtype=torch.uint8, device="cuda") for w in (256, so))
    onorm = (rand(1, kbh, n, 32) * 4).half()
    knorm = (onorm.float() + rand(1, kbh, n, 32) * 6).half()
    idx = rand(1, kbh, n, 128).topk(32, -1)[1].to(torch.uint8)
    qs = (q.float().view(-1, 128) @ S).view(1, kbh * rep, 1, 256) if given else None
    args = (bits, obits, knorm, onorm, idx, qs, q, S)
    got = ops.qjl_gqa_score(*args).cpu()
    for _ in range(3):
        assert torch.equal(ops.qjl_gqa_score(*args).cpu(), got)
    ref = _exact(*[None if t is None else t.cpu() for t in args])
    assert rel_l2(got, ref) <= 1e-5
    err, size = (got.double() - ref).view(kbh, rep, n, 32).norm(dim=-1), ref.view(kbh, rep, n, 32).norm(dim=-1)
    assert float((err / size).max()) <= 4e-5          # group by group
    assert lib().cq_qjl_status() == 0


def test_other_heads_keep_their_scores():
    """A query that is not finite leaves the other heads of its KV head alone."""
    from calibquant_b200 import ops
    g = torch.Generator().manual_seed(5)
    S, q = torch.randn(128, 256, generator=g), torch.randn(1, 4, 1, 128, generator=g).half()
    bits, obits = (torch.randint(0, 256, (1, 1, 5, 32, 32), generator=g, dtype=torch.uint8) for _ in range(2))
    knorm, onorm = (torch.rand(1, 1, 5, 32, generator=g) + 3).half(), torch.rand(1, 1, 5, 32, generator=g).half()
    idx = torch.stack([torch.randperm(128, generator=g)[:32] for _ in range(5)]).view(1, 1, 5, 32).to(torch.uint8)
    args = [t.cuda() for t in (bits, obits, knorm, onorm, idx)]
    base = ops.qjl_gqa_score(*args, None, q.cuda(), S.cuda())
    q[0, 2, 0, 7] = float("inf")
    got = ops.qjl_gqa_score(*args, None, q.cuda(), S.cuda())
    assert torch.equal(got[:, [0, 1, 3]], base[:, [0, 1, 3]]) and not torch.isfinite(got[:, 2]).any()


def _one(dtype, S, q, seed=3, n=9, oc=32, onorm_is=None, knorm_is=None, given=None):
    """(arguments, exact scores) of one KV head's queries q over n groups."""
    g = torch.Generator().manual_seed(seed)
    bits, obits = (torch.randint(0, 256, (1, 1, n, 32, 32), generator=g, dtype=torch.uint8) for _ in range(2))
    onorm = torch.rand(1, 1, n, 32, generator=g).to(dtype) if onorm_is is None else torch.full((1, 1, n, 32), onorm_is, dtype=dtype)
    knorm = (torch.rand(1, 1, n, 32, generator=g) + 3).to(dtype) if knorm_is is None else torch.full((1, 1, n, 32), knorm_is, dtype=dtype)
    idx = torch.stack([torch.randperm(128, generator=g)[:oc] for _ in range(n)]).view(1, 1, n, oc).to(torch.uint8)
    return [bits, obits, knorm, onorm, idx, given, q.to(dtype), S]


def _error(args):
    from calibquant_b200 import ops
    got = ops.qjl_gqa_score(*[None if t is None else t.cuda() for t in args]).cpu()
    return rel_l2(got, _exact(*args))


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -10])
@pytest.mark.parametrize("given", [False, True])
def test_channels_named_many_times(scale, given):
    """Three and more mentions of an fp16 element have more bits than fp16, and with a small projection more than its range.  The
    projection is fp16, so that only sums round."""
    g = torch.Generator().manual_seed(11)
    S, q = (torch.randn(128, 256, generator=g) * scale).half().float(), torch.randn(1, 4, 1, 128, generator=g)
    args = _one(torch.half, S, q, given=None if not given else (q.half().float() @ S))
    idx = args[4]
    idx[:, :, 0, 1:3] = idx[:, :, 0, :1]
    idx[:, :, 4, 5:12] = idx[:, :, 4, :1]
    idx[:, :, 5] = idx[:, :, 5, :1]             # one channel, 32 times
    idx[:, :, 8, 20:] = idx[:, :, 8, :12]       # twelve channels twice
    assert _error(args) <= 1e-5


@pytest.mark.parametrize("dtype", [torch.half, torch.bfloat16])
def test_given_sketch_of_another_size(dtype):
    """The sketch of the query is an argument of its own: larger than the query and the projection let expect, and of a zero query."""
    g = torch.Generator().manual_seed(12)
    S, q = torch.randn(128, 256, generator=g), torch.randn(1, 4, 1, 128, generator=g)
    q[:, 1] = 0
    given = torch.randn(1, 4, 1, 256, generator=g) * torch.tensor([3e4, 10., 3e4, 1.]).view(1, 4, 1, 1)
    args = _one(dtype, S, q, given=given)
    for head in range(4):
        one = args[:5] + [given[:, head:head + 1], args[6][:, head:head + 1], S]
        assert _error(one) <= 1e-5
    assert _error(args) <= 1e-5


def test_bfloat16_queries_near_the_end_of_the_range():
    """128 channels of such numbers are past fp32's range, their scores with small keys are not."""
    g = torch.Generator().manual_seed(13)
    S, q = torch.randn(128, 256, generator=g), torch.randn(1, 4, 1, 128, generator=g) * 1e37
    assert _error(_one(torch.bfloat16, S, q, onorm_is=2.0 ** -9, knorm_is=2.0 ** -8)) <= 1e-5
    assert _error(_one(torch.bfloat16, S, q * 1e-70, onorm_is=1., knorm_is=2.)) <= 1e-5


@pytest.mark.parametrize("given", [False, True])
def test_inlier_part_of_a_query_in_the_outlier_channels(given):
    """Outlier norms of zero: what counts is q S - q_out S, 1/170 of either.  Eight additions of the hi rows' products lose 2^-24 of them
    each in the mean: 8 x 170 x 2^-24 (where the lo rows' follow, sixteen)."""
    g = torch.Generator().manual_seed(14)
    S, q = torch.randn(128, 256, generator=g), torch.randn(1, 4, 1, 128, generator=g)
    q[..., :32] *= 300
    args = _one(torch.half, S, q, onorm_is=0., knorm_is=3., given=None if not given else (q.half().double() @ S.double()).float())
    args[4][...] = torch.arange(32, dtype=torch.uint8)
    assert _error(args) <= 8.2e-5


def test_small_projection():
    """Elements of 1e-3 are kept to 2^-25, 1.7e-5 of them in the mean; a sum of theirs is off by as much."""
    g = torch.Generator().manual_seed(15)
    S, q = torch.randn(128, 256, generator=g) * 1e-3, torch.randn(1, 4, 1, 128, generator=g)
    assert _error(_one(torch.half, S, q, n=60)) <= 2.1e-5


def test_device_status_covers_the_scores(monkeypatch):
    """No wait is made to run out: the library's answer is replaced on the host."""
    from calibquant_b200 import _lib, ops

    class TimedOut:
        cq_qjl_status = staticmethod(lambda: _lib.CQ_ERR_TIMEOUT)

    assert ops.device_status() == 0
    monkeypatch.setattr(ops, "lib", TimedOut)
    assert ops.device_status() == _lib.CQ_ERR_TIMEOUT
