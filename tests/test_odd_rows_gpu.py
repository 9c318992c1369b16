"""Pointwise groups over rows of no whole number of vectors: gathered rows, per-column and per-row operands,
permuted and sliced rows.  Moved values and single rounded operations: exact."""
import pytest
import torch

import inductor_x_b200  # noqa: F401

pytestmark = pytest.mark.gpu


def compiled(fn, *args):
    torch._dynamo.reset()
    return torch.compile(fn, dynamic=False)(*args)


def data(cuda, shape, dtype):
    return torch.randn(*shape, generator=torch.Generator(device=cuda).manual_seed(sum(shape)), device=cuda).to(dtype)


# rows of four vectors and one element, one element short of a vector, short of the length that is taken, long
@pytest.mark.parametrize("dtype,cols", [(torch.float32, 17), (torch.bfloat16, 39), (torch.float16, 15), (torch.bfloat16, 333), (torch.float32, 1023)])
def test_gathered_rows(cuda, dtype, cols):
    table = data(cuda, (301, cols), dtype)
    for n in (1, 777):
        idx = torch.randint(-301, 301, (n,), generator=torch.Generator(device=cuda).manual_seed(n), device=cuda)
        assert torch.equal(compiled(lambda t, i: t[i], table, idx), table[idx])
    flat = data(cuda, (table.numel() + 1,), dtype)
    off = flat[1:].view(table.shape)      # base off a boundary
    assert torch.equal(compiled(lambda t, i: t[i], off, idx), off[idx])


def test_the_template_is_the_one_that_runs(cuda):
    from torch._inductor.utils import run_and_get_code

    torch._dynamo.reset()
    x, w = data(cuda, (9, 333), torch.float16), data(cuda, (333,), torch.float16)
    _, code = run_and_get_code(torch.compile(lambda x, w: torch.maximum(x, w), dynamic=False), x, w)
    assert "launch_pointwise_rows<Body, 333>" in "\n".join(code)


def test_operands_of_rows(cuda):
    x, w, r = data(cuda, (57, 333), torch.bfloat16), data(cuda, (333,), torch.bfloat16), data(cuda, (57, 1), torch.bfloat16)
    assert torch.equal(compiled(lambda x, w, r: torch.maximum(torch.minimum(x, w), r), x, w, r), torch.maximum(torch.minimum(x, w), r))
    assert torch.equal(compiled(lambda x, w: torch.maximum(x, w).float(), x[1:], w), torch.maximum(x[1:], w).float())
    assert torch.equal(compiled(lambda x: (x[:, 3:300] * 2).repeat(1, 2), x), (x[:, 3:300] * 2).repeat(1, 2))
    y = data(cuda, (5, 6, 7, 45), torch.float16)
    assert torch.equal(compiled(lambda y: (y.permute(2, 0, 1, 3) * 2).contiguous(), y), y.permute(2, 0, 1, 3) * 2)
    buf = torch.full((x.numel() + 64,), 7.0, dtype=x.dtype, device=cuda)
    out = buf[33:33 + x.numel()].view(x.shape)   # results off a boundary, in a larger buffer
    compiled(lambda x, w, out: out.copy_(torch.maximum(x, w)), x, w, out)
    assert torch.equal(out, torch.maximum(x, w)) and bool((buf[:33] == 7).all()) and bool((buf[33 + x.numel():] == 7).all())


# whole numbers: the sums are exact in any order
@pytest.mark.parametrize("dtype,cols", [(torch.float32, 333), (torch.bfloat16, 2053)])
def test_rows_beside_masked_loads_and_atomic_sums(cuda, dtype, cols):
    from torch._inductor.utils import run_and_get_code

    g = torch.Generator(device=cuda).manual_seed(cols)
    t, y = (torch.randint(-4, 5, (n, c), generator=g, device=cuda).to(dtype) for n, c in ((61, cols), (77, cols - 3)))
    i, j = (torch.randint(0, n, (77,), generator=g, device=cuda) for n in (61, 9))

    def padded(t, i, y):
        return torch.maximum(t[i], torch.nn.functional.pad(y, (3, 0)))

    def summed(t, i, j):
        return torch.zeros(9, cols, device=t.device, dtype=torch.float32).index_add(0, j, t[i].float())

    for fn, args in ((summed, (t, i, j)), (padded, (t, i, y)))[:1 if cols == 333 else 2]:   # (short rows beside a mask are not)
        torch._dynamo.reset()
        got, code = run_and_get_code(torch.compile(fn, dynamic=False), *args)
        assert torch.equal(got, fn(*args))
        assert f"launch_pointwise_rows<Body, {cols}>" in "\n".join(code)
