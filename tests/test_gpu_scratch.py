"""Scratch of the decode steps under CUDA graphs: a graph keeps the buffer that it was captured with, whatever larger steps and
other captures ask for afterwards on the same stream."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(B, t_vis, seed):
    from calibquant_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(seed)
    k, v = (torch.randn(B, 8, t_vis, 128, generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn(B, 32, 1, 128, generator=g, device="cuda").half()
    packs = ops.pack_k_per_channel(k, 32, 1), ops.pack_v_per_token(v, 32, 1)
    return lambda: ops.decode_attention(q, *packs, None, None, 0, 1)


def _capture(step, side, warm):
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        if warm:
            step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = step()
    return graph, out


def _scratch(side):
    from calibquant_b200._lib import native
    return native().workspaces_of(torch.cuda.current_device(), side.cuda_stream)


@pytest.mark.parametrize("warm", [True, False])
def test_graph_keeps_its_scratch(warm):
    small, large = _step(1, 65536, 1), _step(2, 131072, 2)      # several launches each: logits and partial sums in the scratch
    want = small()
    side = torch.cuda.Stream()
    graph, out = _capture(small, side, warm)
    with torch.cuda.stream(side):
        want_large = large()                                    # a larger step on the same stream takes a larger buffer
    torch.cuda.synchronize()
    other, out_large = _capture(large, side, False)
    # whatever was given back is handed out here
    fills = [torch.full((1 << 18,), i % 251, dtype=torch.uint8, device="cuda") for i in range(256)]
    for i in range(3):
        graph.replay()
        other.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(out_large, want_large)
    assert all(bool((f == i % 251).all()) for i, f in enumerate(fills))


def test_retired_scratch_is_bounded():
    """A buffer that a graph has used is replaced by one of at least twice its size; others grow to what is asked for."""
    from calibquant_b200._lib import native
    side, dev = torch.cuda.Stream(), torch.cuda.current_device()
    with torch.cuda.stream(side):
        assert native().workspace(1000, dev, side.cuda_stream).numel() == 1000
        assert native().workspace(1100, dev, side.cuda_stream).numel() == 1100
    torch.cuda.synchronize()
    graph, x = torch.cuda.CUDAGraph(), torch.zeros(1, device="cuda")
    with torch.cuda.graph(graph, stream=side):
        x.add_(1)
        assert native().workspace(1050, dev, side.cuda_stream).numel() == 1100
    with torch.cuda.stream(side):
        assert native().workspace(1200, dev, side.cuda_stream).numel() == 2200
    assert [b.numel() for b in _scratch(side)] == [2200]
