"""Other Python threads go on while a thread waits to launch: the entry points give the interpreter up for the C call."""

import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_interpreter_is_free_while_a_launch_waits():
    from calibquant_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(0)
    k = torch.randn(1, 2, 64, 128, generator=g, device="cuda").half()
    q, fp = torch.randn(1, 8, 1, 128, generator=g, device="cuda").half(), k[:, :, :8].contiguous()
    packs = ops.pack_k_per_channel(k, 32, 1), ops.pack_v_per_token(k, 32, 1)
    want = ops.decode_attention(q, *packs, fp, fp, 4, 1)
    torch.cuda.synchronize()
    started, result = threading.Event(), []

    def issue():
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(1_200_000_000)      # ~0.6 s of the SM clock; the stream's queue fills up behind it
            started.set()
            t = time.perf_counter()
            for _ in range(4000):
                out = ops.decode_attention(q, *packs, fp, fp, 4, 1)
            torch.cuda.current_stream().synchronize()
            result.extend([out, time.perf_counter() - t])

    worker = threading.Thread(target=issue)
    worker.start()
    started.wait()
    gap, last = 0.0, time.perf_counter()
    while worker.is_alive():
        time.sleep(0.002)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    worker.join()
    assert torch.equal(result[0], want)
    assert result[1] > 0.3 and gap < 0.2, (result[1], gap)
