"""A normalisation layer's training step through plain ``torch.compile``: its backward sums over rows
(the statistic's gradient) and over columns (the weight's), which this backend keeps apart."""
import pytest
import torch
import torch.nn.functional as F

from inductor_x_b200.llama_layer import rms_norm


def rms(x, w):
    return rms_norm(x, w, 1e-6)


def layer(x, w):
    return F.layer_norm(x, (x.shape[-1],), w, None, 1e-5)


def test_fusion_of_the_two_orders_is_off():
    import inductor_x_b200  # noqa: F401
    from torch._inductor import config

    assert config.triton.mix_order_reduction is False


# the smaller one is below the size from which Inductor mixes the orders, the others are above it
@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(300, 257), (8192, 2048), (33000, 1111)])
@pytest.mark.parametrize("fn", [rms, layer])
def test_gradients(cuda, fn, rows, cols):
    g = torch.Generator(device=cuda).manual_seed(rows)
    x, dy = (torch.randn(rows, cols, generator=g, device=cuda).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(cols, generator=g, device=cuda)).bfloat16()
    got, want = [], []
    torch._dynamo.reset()
    for f, wide, into in ((torch.compile(fn, dynamic=False), lambda t: t, got), (fn, lambda t: t.double(), want)):
        xs, ws = (wide(t).detach().clone().requires_grad_(True) for t in (x, w))
        y = f(xs, ws)
        into += [y.detach(), *torch.autograd.grad(y, (xs, ws), wide(dy))]
    for a, b in zip(got, want):
        # 32-bit sums rounded once to bf16: two roundings of the type, against the root mean square
        err = (a.double() - b).abs() / b.abs().clamp_min(float(b.square().mean().sqrt()))
        assert float(err.max()) <= 8e-3
