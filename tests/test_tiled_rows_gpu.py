"""Short rows of a permuted view, walked in 16 x 16 tiles: row counts below, at and just above one
batch for every resident block, where the batches turn from strided to consecutive, and a last
batch that is not full.  Sums of 16-bit values in 32 bits, rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shape", [(torch.float16, (1, 16, 16, 64)), (torch.bfloat16, (37, 64, 128, 64)),
                                         (torch.float16, (21, 128, 256, 32)), (torch.float32, (19, 112, 144, 64)),
                                         (torch.float16, (64, 128, 256, 64))])
def test_sum_of_short_rows(cuda, dtype, shape):
    import inductor_x_b200  # noqa: F401
    from torch._inductor.utils import run_and_get_code

    g = torch.Generator(device=cuda).manual_seed(sum(shape))
    x = torch.rand(*shape, generator=g, device=cuda).to(dtype)
    torch._dynamo.reset()
    out, code = run_and_get_code(torch.compile(lambda t: t.permute(0, 2, 1, 3).sum(3), dynamic=False), x)
    assert "kTiled = true" in "\n".join(code)
    want = x.permute(0, 2, 1, 3).double().sum(3)
    tol = {torch.float32: 1e-5, torch.float16: 1e-3, torch.bfloat16: 8e-3}[dtype]
    assert float(((out.double() - want).abs() / want.abs()).max()) <= tol
