"""A column reduction whose terms carry a per-row statistic (a weight gradient: the sum over the
tokens of dy * x * rstd[token]): the statistic is stride-1 along the reduced axis but does not
depend on the kept one, so the group is an outer reduction with one scalar a step."""
import pytest
import torch


def weight_grad(dy, x, rstd):
    return (dy.float() * (x.float() * rstd[:, None])).sum(0).to(x.dtype)


def scaled_max(dy, x, rstd):
    return (x * rstd[:, None] + dy).amax(0)


FORMS = [(weight_grad, torch.bfloat16, 4096, 1024), (weight_grad, torch.float16, 333, 77), (scaled_max, torch.float32, 1000, 64),
         (weight_grad, torch.float32, 40, 2056)]


def make(rows, cols, dtype, device):
    g = torch.Generator().manual_seed(rows + cols)
    dy, x = (torch.randn(rows, cols, generator=g).to(dtype).to(device) for _ in range(2))
    return dy, x, (0.5 + torch.rand(rows, generator=g)).to(device)


@pytest.mark.parametrize("fn,dtype,rows,cols", FORMS)
def test_taken_as_an_outer_reduction(dry_backend, fn, dtype, rows, cols):
    from torch._inductor.utils import run_and_get_code

    torch._dynamo.reset()
    _, code = run_and_get_code(torch.compile(fn, dynamic=False), *make(rows, cols, dtype, "cpu"))
    text = "\n".join(code)
    assert "ld_uniform(" in text and ("launch_outer_gen<" in text or "launch_outer_split_gen<" in text)


@pytest.mark.parametrize("form", ["row operand", "both"])
def test_row_operands_stay_rows(dry_backend, form):
    """A load that depends on both axes and is stride-1 along the reduced one is a row, whatever
    stands beside it."""
    from torch._inductor.utils import run_and_get_code

    def f(a, s):
        return (a * s).sum(1)

    def g(a, b, s):
        return (a * b.t() * s).sum(1)

    a, b, s = torch.randn(96, 256), torch.randn(256, 96), torch.randn(256)
    torch._dynamo.reset()
    _, code = run_and_get_code(torch.compile(f if form == "row operand" else g, dynamic=False),
                               *((a, s) if form == "row operand" else (a, b, s)))
    assert "launch_row_gen<" in "\n".join(code)


@pytest.mark.gpu
@pytest.mark.parametrize("fn,dtype,rows,cols", FORMS)
def test_against_64_bits(cuda, fn, dtype, rows, cols):
    import inductor_x_b200  # noqa: F401

    args = make(rows, cols, dtype, cuda)
    torch._dynamo.reset()
    got = torch.compile(fn, dynamic=False)(*args)
    want = fn(*(t.double() for t in args))
    # sums of `rows` terms of either sign: the bound is relative to the root mean square
    tol = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}[dtype]
    err = (got.double() - want.double()).abs() / want.double().abs().clamp_min(float(want.double().square().mean().sqrt()))
    assert float(err.max()) <= tol


def test_sum_over_many_rows_with_a_statistic_is_an_outer_reduction(dry_backend):
    """More rows than one block could hold as a row: the statistic's stride of 1 along them does not make
    the group a row walked in chunks (100000 x 1024: 870 us that way against 90)."""
    from torch._inductor.utils import run_and_get_code

    torch._dynamo.reset()
    x, dy = (torch.empty(70000, 64, dtype=torch.bfloat16) for _ in range(2))
    fn = lambda x, dy, rstd: (dy.float() * x.float() * rstd).sum(0)
    code = "\n".join(run_and_get_code(torch.compile(fn, dynamic=False), x, dy, torch.empty(70000, 1))[1])
    assert "launch_outer" in code and "launch_row_gen" not in code
