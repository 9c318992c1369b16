"""The attention kernels called from threads that have not used the device before: all memory comes out of the
allocator's cache, so nothing but these calls brings the thread a context."""
import threading

import pytest
import torch

from inductor_x_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("direction", ["forward", "backward"])
def test_first_call_of_a_thread(cuda, direction):
    q, k, v, dy = (torch.randn(1, 2, 130, 128, device=cuda).half() for _ in range(4))
    out, lse = ops.fused_attention(q, k, v, 0.1, return_lse=True)

    def call():
        if direction == "forward":
            return ops.fused_attention(q, k, v, 0.1, return_lse=True)
        return ops.fused_attention_backward(q, k, v, out, lse, dy, 0.1)

    def work():
        try:
            got.append(call())
        except Exception as e:  # noqa: BLE001 - asserted below, in the test's own thread
            got.append(e)

    got = [call()]
    want = [t.clone() for t in got.pop()]  # and the results' own memory is in the cache again
    torch.cuda.synchronize()
    thread = threading.Thread(target=work)
    thread.start()
    thread.join(60)
    assert got and not isinstance(got[0], Exception), got
    torch.cuda.synchronize()
    for a, b in zip(got[0], want):
        assert torch.equal(a, b)
