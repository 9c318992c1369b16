"""Gradients of the compact attention op when one of its two outputs has none: that of the log-sum-exp is never
read, so nothing is made for it; without one of the output the gradients are zero, as they were."""
import pytest
import torch

import inductor_x_b200.fusion_attention_graph  # noqa: F401  (registers the op)
from torch.fx.experimental.proxy_tensor import make_fx


def _inputs(device):
    return [torch.randn(1, 2, 130, 128, device=device, dtype=torch.float16, requires_grad=True) for _ in range(3)]


def test_no_zeros_for_the_log_sum_exp():
    q, k, v = _inputs("meta")

    def step(q, k, v, dy):
        out, _ = torch.ops.b200_graph.b200_sdpa(q, k, v, 0.1, True)
        return torch.autograd.grad(out, (q, k, v), dy)

    ops = [str(n.target) for n in make_fx(step, tracing_mode="fake")(q, k, v, torch.empty_like(q)).graph.nodes]
    assert any("b200_sdpa_backward" in n for n in ops) and not any("zeros" in n for n in ops)


@pytest.mark.gpu
@pytest.mark.parametrize("used", ["out", "lse", "both"])
def test_gradients_of_each_output(cuda, used):
    leaves = _inputs(cuda)
    out, lse = torch.ops.b200_graph.b200_sdpa(*leaves, 0.1, True)
    outputs = {"out": (out,), "lse": (lse,), "both": (out, lse)}[used]
    got = torch.autograd.grad(outputs, leaves, [torch.ones_like(t) for t in outputs])
    dy = torch.zeros_like(out) if used == "lse" else torch.ones_like(out)
    want = torch.ops.b200_graph.b200_sdpa_backward(*(t.detach() for t in (*leaves, out, lse)), dy, 0.1, True)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
        assert used != "lse" or not a.any()
