"""Sums that ride in the softmax exchange, on rows that do not fill their threads' vectors: the
weight of such a sum is computed for the elements past the end of the row too, from zeros, and a
reciprocal or a logarithm of those is not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def weighted(x, y):
    r = 1.0 / y
    return (torch.softmax(x * r, -1) * r).sum(-1)


# teams of a part of a warp, a warp, and several; 1024 fills its vectors
@pytest.mark.parametrize("cols", [37, 100, 1000, 1003, 1024, 2500])
def test_weights_past_the_end_of_the_row(cuda, cols):
    import inductor_x_b200  # noqa: F401
    from torch._inductor.utils import run_and_get_code

    g = torch.Generator(device=cuda).manual_seed(cols)
    x, y = torch.randn(64, cols, generator=g, device=cuda), 1 + torch.rand(64, cols, generator=g, device=cuda)
    torch._dynamo.reset()
    out, code = run_and_get_code(torch.compile(weighted, dynamic=False), x, y)
    assert "online_softmax<1, 0, true>" in "\n".join(code)
    torch.testing.assert_close(out.double(), weighted(x.double(), y.double()), rtol=1e-5, atol=0)
