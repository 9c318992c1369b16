"""Transposes by way of shared memory: extents that register tiles do not divide, rows off a 16-byte boundary on
either side.  Moved values and one rounded addition: exact."""
import pytest
import torch

import inductor_x_b200  # noqa: F401

pytestmark = pytest.mark.gpu


def compiled(fn, *args):
    torch._dynamo.reset()
    return torch.compile(fn, dynamic=False)(*args)


def data(cuda, shape, dtype):
    return torch.randn(*shape, generator=torch.Generator(device=cuda).manual_seed(sum(shape)), device=cuda).to(dtype)


# extents around 32 (the shortest taken), a block's columns (60 and 120, one and two of them) and its vectors
# of an output row (64 and 128 elements, less what a row's start off a boundary takes)
@pytest.mark.parametrize("dtype,b,c", [(torch.float16, 32, 33), (torch.float16, 58, 121), (torch.float16, 129, 240), (torch.bfloat16, 700, 131),
                                       (torch.float32, 33, 32), (torch.float32, 121, 61), (torch.float32, 65, 120)])
def test_extents(cuda, dtype, b, c):
    x = data(cuda, (3, b, c), dtype)
    assert torch.equal(compiled(lambda x: (x.transpose(1, 2) + 1.0).contiguous(), x), x.transpose(1, 2) + 1.0)


def test_the_template_is_the_one_that_runs(cuda):
    from torch._inductor.utils import run_and_get_code

    torch._dynamo.reset()
    x = data(cuda, (2, 65, 59), torch.float16)
    _, code = run_and_get_code(torch.compile(lambda x: (x.transpose(1, 2) + 1.0).contiguous(), dynamic=False), x)
    assert "launch_pointwise_smem" in "\n".join(code)


def test_groups(cuda):
    """Digits between and beyond the two, a second operand of the same order, one of the output's order and one
    that is constant along rows, results of another width, operands and results off a boundary."""
    dtype = torch.bfloat16
    x, y = data(cuda, (3, 37, 5, 61), dtype), data(cuda, (3, 37, 5, 61), dtype)
    w, z = data(cuda, (61, 1), dtype), data(cuda, (3, 5, 61, 37), dtype)
    for order in ((0, 3, 1, 2), (0, 2, 3, 1)):
        assert torch.equal(compiled(lambda x: (x.permute(order) * 2).contiguous(), x), x.permute(order) * 2)
    assert torch.equal(compiled(lambda x, y: torch.maximum(x.permute(0, 2, 3, 1), y.permute(0, 2, 3, 1)).contiguous(), x, y),
                       torch.maximum(x, y).permute(0, 2, 3, 1))
    assert torch.equal(compiled(lambda x, w, z: torch.maximum(torch.minimum(x.permute(0, 2, 3, 1), w), z).float(), x, w, z),
                       torch.maximum(torch.minimum(x.permute(0, 2, 3, 1), w), z).float())
    flat = data(cuda, (x.numel() + 1,), dtype)
    buf = torch.full((x.numel() + 64,), 7.0, dtype=dtype, device=cuda)
    out = buf[32:32 + x.numel()].view(3, 5, 61, 37)
    for v in (x, flat[1:].view(x.shape)):
        compiled(lambda v, out: out.copy_(v.permute(0, 2, 3, 1)), v, out)
        assert torch.equal(out, v.permute(0, 2, 3, 1)) and bool((buf[:32] == 7).all()) and bool((buf[32 + x.numel():] == 7).all())
    part = data(cuda, (40, 3, 90), dtype)[:, :, 7:80]   # a view with a pitch
    assert torch.equal(compiled(lambda p: (p.transpose(0, 2) + 1).contiguous(), part), part.transpose(0, 2) + 1)


def test_three_operands_keep_the_gathers(cuda):
    x, y, z = (data(cuda, (2, 45, 67), torch.float16) for i in range(3))
    got = compiled(lambda x, y, z: torch.maximum(torch.maximum(x.transpose(1, 2), y.transpose(1, 2) * 2), z.transpose(1, 2) * 3).contiguous(), x, y, z)
    assert torch.equal(got, torch.maximum(torch.maximum(x, y * 2), z * 3).transpose(1, 2))
