"""Reductions over teams of one to 32 warps: what warps exchange is read by every thread (softmax up to four warps,
sums from four to sixteen) or folded by shuffles.  Against 64-bit arithmetic, rows with one dominant element in
each warp's part, rows of the lowest value and of infinities among them."""
import pytest
import torch

import inductor_x_b200  # noqa: F401

pytestmark = pytest.mark.gpu


# fp32 rows of 64, 128, 256 and 1024 threads of two vectors
@pytest.mark.parametrize("cols", [512, 1024, 2048, 8192])
def test_teams(cuda, cols):
    g = torch.Generator(device=cuda).manual_seed(cols)
    x = torch.randn(300, cols, generator=g, device=cuda)
    x[:128, :] = -3e38
    x[torch.arange(128), torch.arange(128) * (cols // 128)] = 3e38    # the maximum in each part of the row
    x[128, :], x[129, : cols // 2], x[130, 1:] = -3.4028234e38, float("-inf"), float("-inf")
    gain = torch.randn(cols, generator=g, device=cuda)

    def chain(x, gain):     # the maximum, the sum, a sum of exponentials times a weight and a plain sum in one exchange
        y = torch.softmax(x, -1) * gain
        return torch.softmax(x, -1), y.mean(-1), x.abs().clamp(max=10).sum(-1), x.amax(-1)

    torch._dynamo.reset()
    p, m, s, top = torch.compile(chain, dynamic=False)(x, gain)
    pd, md, sd, td = chain(x.double(), gain.double())
    assert float((p.double() - pd).abs().max()) <= 2e-6
    assert float((m.double() - md).abs().max()) <= 1e-6
    assert float(((s.double() - sd) / sd).abs().max()) <= 1e-5
    assert torch.equal(top, x.amax(-1))
