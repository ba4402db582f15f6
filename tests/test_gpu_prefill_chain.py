"""Launches that come up while the one before them runs: the quantize or pack calls of a prompt and its attention.

Each of them waits for the end of the launch before it.  The same calls with the device synchronised between them have to
give the same bytes, also where the next write of the inputs follows directly (a late reader would see it)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HKV, D, SYS = 8, 128, 41


def _chain(qkv, tables, vis, rep, bits, fmt, between):
    from calibquant_b200 import calibquant, ops
    batch, tokens = qkv.shape[:2]
    k_cache = torch.zeros(batch, HKV, tokens - vis, D, dtype=qkv.dtype, device="cuda")
    v_cache = torch.zeros_like(k_cache)
    q, k, v = ops.prefill_rope_split(qkv, *tables, HKV, rep, k_cache, v_cache, SYS, vis)
    between()
    k_span, v_span = k[:, SYS:SYS + vis], v[:, SYS:SYS + vis]
    if fmt == "uint8":
        packs = list(calibquant.quant_encode(k_span, bits))
        between()
        packs += calibquant.quant_encode(v_span, bits)
    else:
        packs = list(ops.pack_k_per_channel(k_span.transpose(1, 2), 32, bits))
        between()
        packs += ops.pack_v_per_token(v_span.transpose(1, 2), 32, bits)
    between()
    out = ops.prefill_attention(q, k, v)
    between()
    for x in (qkv, q, k, v):                   # directly behind the readers
        x.fill_(float("nan"))
    return [out, *packs, k_cache, v_cache]


@pytest.mark.parametrize("fmt", ["uint8", "group"])
@pytest.mark.parametrize("batch,vis,rep,bits,dtype", [
    (1, 32, 4, 1, torch.bfloat16),             # one CTA a head
    (2, 1280, 4, 2, torch.float16),            # clusters of 8, rows kept in registers
    (1, 2528, 6, 4, torch.bfloat16),           # the last slice ragged, rows read twice
    (48, 288, 4, 2, torch.bfloat16),           # more CTAs than fit at once
])
def test_chain_as_if_synchronised(batch, vis, rep, bits, dtype, fmt):
    tokens = SYS + vis + 23
    g = torch.Generator(device="cuda").manual_seed(vis)
    first = torch.randn(batch, tokens, HKV * (rep + 2) * D, generator=g, device="cuda").to(dtype)
    angle = torch.rand(tokens, D, generator=g, device="cuda") * 6.28
    tables = (angle.cos().to(dtype), angle.sin().to(dtype), torch.arange(tokens, device="cuda")[None].expand(batch, tokens).contiguous())
    want = _chain(first.clone(), tables, vis, rep, bits, fmt, torch.cuda.synchronize)
    torch.cuda.synchronize()
    x = torch.empty_like(first)

    def again():
        x.copy_(first)
        return _chain(x, tables, vis, rep, bits, fmt, lambda: None)

    runs = [again() for _ in range(8)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        again()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = again()
    for _ in range(4):
        graph.replay()
    torch.cuda.synchronize()
    for got in runs + [captured]:
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
