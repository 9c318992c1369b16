"""Softmax of rows masked with the lowest value of their type (not -inf): what a row's largest value times log2 e
cannot be held in."""
import pytest
import torch

# exp and the quotient in fp32, rounded once
TOL = {torch.float32: 1e-5, torch.bfloat16: 1.6e-2}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cols", [40, 64, 1537, 4096, 70000, 131072 + 8])
def test_masked_rows(cuda, dtype, cols):
    """Sub-warp teams, odd rows, whole teams, rows walked in chunks; the second half, everything and everything
    but one element at the lowest value, and the largest value in one place."""
    import inductor_x_b200  # noqa: F401

    g = torch.Generator(device=cuda).manual_seed(cols)
    lim = torch.finfo(dtype)
    x = torch.randn(40, cols, generator=g, device=cuda).to(dtype)
    x[0:8, cols // 2:] = lim.min
    x[8:16] = lim.min
    x[16:24, 1:] = lim.min
    x[24:32, :-1] = lim.min
    x[32, 3] = lim.max
    x[33, cols // 3:] = float("-inf")
    want = x.double().softmax(-1)
    forms = (lambda x: x.softmax(-1), lambda x: torch.log_softmax(x, -1).exp(), lambda x: (x - x.amax(-1, keepdim=True)).float().exp())
    for fn in forms if cols == 4096 else forms[:1]:
        torch._dynamo.reset()
        got = torch.compile(fn, dynamic=False)(x).double()
        if fn(torch.zeros(1, 2))[0, 0] == 1:
            got = got / got.sum(-1, keepdim=True)
        assert bool(got.isfinite().all())
        assert float(((got - want).abs() / want.clamp_min(float(want.square().mean().sqrt()))).max()) <= TOL[dtype]
