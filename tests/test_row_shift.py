"""Generated row kernels whose blocks keep to one offset from the 16-byte boundaries (kShiftPeriod)."""
import re
import shutil

import pytest
import torch
import torch.nn.functional as F

needs_nvcc = pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")


def chain(x, g, gamma, beta):
    return F.layer_norm(torch.softmax(x, -1) * g + x, (x.shape[-1],), gamma, beta, 1e-5)


def _period(fn, *args):
    """(period, row_offset) of the module, period 0 where its rows are shifted one by one."""
    from torch._inductor.utils import run_and_get_code

    torch._dynamo.reset()
    code = "\n".join(run_and_get_code(torch.compile(fn, dynamic=False), *args)[1])
    assert code.count("ixb_load_kernel('''") == 1
    period = int(re.search(r"kShiftPeriod = (\d+);", code).group(1))
    expr = re.search(r"row_offset\(int x\) const \{ return \(int\)\((.*?)\); \}", code).group(1)
    return period, lambda x: eval(expr.replace("(long long)", ""), {"x": x}), code


@needs_nvcc
@pytest.mark.parametrize("dtype,cols,pitch,first", [
    (torch.float16, 1537, 1537, 0), (torch.bfloat16, 515, 518, 0), (torch.float32, 1030, 1030, 0), (torch.float32, 1031, 1033, 2),
    (torch.float16, 1537, 1600, 3), (torch.float16, 1540, 1544, 0)])
def test_rows_a_period_apart_lie_alike(dry_backend, dtype, cols, pitch, first):
    x = torch.randn(40 * pitch + first).to(dtype)[first:].view(40, pitch)[:, :cols]
    p = [torch.randn(cols).to(dtype) for _ in range(2)]
    # (the result has rows of its own: it takes part with a pitch of `cols`, so the sum alone is looked at)
    period, offset, code = _period(lambda x, g, b: (x * g + b).square().sum(-1), x, *p)
    vec = 16 // x.element_size()
    assert period > 0 and vec % period == 0
    for row in range(3 * vec):       # against the addresses themselves (the view's base counts as aligned)
        assert offset(row % period) == (row * pitch) % vec
    assert "RawRowU" not in code


@needs_nvcc
def test_rows_of_several_pitches_are_shifted_one_by_one(dry_backend):
    x = torch.randn(40, 1544).half()[:, :1537]            # aligned rows in, odd rows out
    p = [torch.randn(1537).half() for _ in range(3)]
    period, _, code = _period(chain, x, *p)
    assert period == 0 and "RawRowU" in code and "put_row_any" in code
    period, _, _ = _period(lambda x: x.cumsum(-1), torch.randn(40, 1537).half())
    assert period == 0                                     # a scan
    period, _, _ = _period(lambda x: x.float().sum(-1), torch.randn(40, 33).half())
    assert period == 0                                     # teams narrower than a warp


TOL = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def _close(got, want, dtype):
    err = (got.double() - want).abs() / want.abs().clamp_min(float(want.square().mean().sqrt()))
    assert float(err.max()) <= TOL[dtype]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 257), (3, 511), (7, 1021), (9, 2047), (2000, 1537), (17, 2049), (40, 4099), (5, 8191)])
def test_chain_of_odd_rows(cuda, dtype, rows, cols):
    """Fewer rows than offsets, one element past a vector, one short of it, rows in the middle of a
    buffer that is not to be written beside them."""
    import inductor_x_b200  # noqa: F401

    g = torch.Generator(device=cuda).manual_seed(cols)
    x = torch.randn(rows, cols, generator=g, device=cuda).to(dtype)
    p = [(1 + 0.1 * torch.randn(cols, generator=g, device=cuda)).to(dtype) for _ in range(3)]
    torch._dynamo.reset()
    into = torch.compile(lambda x, g, gamma, beta, out: out.copy_(chain(x, g, gamma, beta)), dynamic=False)
    buf = torch.full((rows * cols + 64,), 7.0, dtype=dtype, device=cuda)
    out = buf[:rows * cols].view(rows, cols)
    into(x, *p, out)
    _close(out, chain(*(t.double() for t in (x, *p))), dtype)
    assert bool((buf[rows * cols:] == 7).all())


@pytest.mark.gpu
def test_other_bodies_of_odd_rows(cuda):
    """In-place rows, three streamed operands of two widths, a mask of bytes, per-row statistics, an
    arg-reduction, operands that are infinite, rows of the lowest values."""
    import inductor_x_b200  # noqa: F401

    g = torch.Generator(device=cuda).manual_seed(3)
    rows, cols = 301, 1283
    x, y, z = (torch.randn(rows, cols, generator=g, device=cuda).half() for _ in range(3))
    f = torch.randn(rows, cols, generator=g, device=cuda)
    m = torch.rand(rows, cols, generator=g, device=cuda) < 0.5
    w = torch.randn(cols, generator=g, device=cuda).half()

    def run(fn, *args):
        torch._dynamo.reset()
        return torch.compile(fn, dynamic=False)(*args)

    a = x.clone()
    run(lambda a: a.add_(a.float().mean(-1, keepdim=True)), a)
    _close(a, x.double() + x.double().mean(-1, keepdim=True), torch.float16)
    _close(run(lambda x, y, z, f, w: (x.float() * y + z * f).softmax(-1) * w, x, y, z, f, w),
           (x.double() * y + z.double() * f.double()).softmax(-1) * w.double(), torch.float32)
    masked = run(lambda f, m: torch.where(m, f, float("-inf")).softmax(-1), f, m)
    _close(masked, torch.where(m, f.double(), float("-inf")).softmax(-1), torch.float32)
    var, mean = run(lambda f: torch.var_mean(f, -1), f)
    _close(var, f.double().var(-1), torch.float32)
    _close(mean, f.double().mean(-1), torch.float32)
    assert torch.equal(run(lambda f: f.argmax(-1), f), f.argmax(-1))
    low = torch.full((9, cols), torch.finfo(torch.float32).min, device=cuda)
    assert torch.equal(run(lambda t: t.amax(-1), low), low.amax(-1))
    assert torch.equal(run(lambda t: (t.softmax(-1) * cols).round(), low * 1e-34), torch.ones_like(low))
    f[5, -1] = float("inf")
    f[7, 0] = float("nan")
    got, want = run(lambda t: t.amax(-1), f), f.amax(-1)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~want.isnan()], want[~want.isnan()])
    inv = run(lambda t: (1 / t).sum(-1), torch.full((9, cols), 2.0, device=cuda))   # 1 / 0 past the ends of a row
    assert torch.equal(inv, torch.full_like(inv, cols / 2))
