"""Rows that start off a 16-byte boundary (odd row lengths, odd offsets and pitches): the staged
covering words, the loads on the spot, the shifted stores and their ends.  Against 64-bit arithmetic
on the same inputs; results are 32-bit sums rounded once, so the bound is a few roundings of the
storage type."""
import pytest
import torch
import torch.nn.functional as F

from inductor_x_b200 import ops

pytestmark = pytest.mark.gpu
TOL = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def chain(x, g, gamma, beta):
    return F.layer_norm(torch.softmax(x, -1) * g + x, (x.shape[-1],), gamma, beta, 1e-5)


def inputs(cuda, rows, cols, dtype, seed=0):
    g = torch.Generator(device=cuda).manual_seed(rows + cols + seed)
    x = torch.randn(rows, cols, generator=g, device=cuda).to(dtype)
    return [x] + [(1 + 0.1 * torch.randn(cols, generator=g, device=cuda)).to(dtype) for _ in range(3)]


def close(got, want, dtype):
    err = (got.double() - want).abs() / want.abs().clamp_min(float(want.square().mean().sqrt()))
    assert float(err.max()) <= TOL[dtype]


# sub-warp teams with several rows in flight, one warp, several warps, two vectors a thread; a row
# that ends one element into a vector, one before its end, and in the middle
SHAPES = [(torch.float16, 301, 33), (torch.bfloat16, 64, 71), (torch.float32, 77, 130), (torch.bfloat16, 9, 515),
          (torch.float16, 1500, 1537), (torch.float32, 5, 3001), (torch.bfloat16, 1, 9001)]


@pytest.mark.parametrize("dtype,rows,cols", SHAPES)
def test_compiled_rows_requested_ahead(cuda, dtype, rows, cols):
    """Every base pointer is 16-byte aligned, so the covering words of a row are fetched while the one
    before it is worked on; an odd length or pitch moves the rows off the boundary.  NaN in the gap
    between rows and behind the last one is not to reach a result."""
    import inductor_x_b200  # noqa: F401

    x, g, gamma, beta = inputs(cuda, rows, cols, dtype)
    want = chain(*(t.double() for t in (x, g, gamma, beta)))
    for pitch in (cols, cols + 4 if cols % 2 else cols + 3):
        torch._dynamo.reset()
        into = torch.compile(lambda x, g, gamma, beta, out: out.copy_(chain(x, g, gamma, beta)), dynamic=False)
        store = torch.full((rows * pitch + 64,), float("nan"), dtype=dtype, device=cuda)
        src = store[:rows * pitch].view(rows, pitch)[:, :cols]
        src.copy_(x)
        buf = torch.full((rows * pitch + 128,), 7.0, dtype=dtype, device=cuda)
        dst = buf[64:64 + rows * pitch].view(rows, pitch)[:, :cols]
        assert all(t.data_ptr() % 16 == 0 for t in (src, g, gamma, beta, dst))
        into(src, g, gamma, beta, dst)
        close(dst, want, dtype)
        dst.fill_(7)  # nothing beyond the rows is written
        assert bool((buf == 7).all())


@pytest.mark.parametrize("dtype,rows,cols", SHAPES)
def test_compiled_rows_inside_a_larger_buffer(cuda, dtype, rows, cols):
    """An output whose base pointer is not 16-byte aligned: rows are loaded when they are worked on."""
    import inductor_x_b200  # noqa: F401

    x, g, gamma, beta = inputs(cuda, rows, cols, dtype)
    torch._dynamo.reset()
    into = torch.compile(lambda x, g, gamma, beta, out: out.copy_(chain(x, g, gamma, beta)), dynamic=False)
    buf = torch.full(((rows + 2) * cols,), 7.0, dtype=dtype, device=cuda)
    into(x, g, gamma, beta, buf[cols:-cols].view(rows, cols))
    want = chain(*(t.double() for t in (x, g, gamma, beta)))
    close(buf[cols:-cols].view(rows, cols), want, dtype)
    assert bool((buf[:cols] == 7).all()) and bool((buf[-cols:] == 7).all())  # nothing beyond the rows is written


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_compiled_rows_of_a_view(cuda, dtype):
    """An odd pitch, an odd first element and per-column operands off a boundary: base pointers that are
    not 16-byte aligned take the loads that are not requested ahead."""
    import inductor_x_b200  # noqa: F401

    x, g, gamma, beta = inputs(cuda, 50, 205, dtype)
    torch._dynamo.reset()
    fn = torch.compile(chain, dynamic=False)
    for view in (x[:, 1:201], x[1:, 3:203]):
        args = [view] + [t[1:201] for t in (g, gamma, beta)]
        close(fn(*args), chain(*(t.double() for t in args)), dtype)


# 12001: rmsnorm holds rows of up to 16384 fp32 columns, and the three per-column operands of
# softmax_layernorm have to fit 227 KB of shared memory in 32 bits (19370 columns)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(3, 1), (7, 33), (200, 515), (2, 9001), (1, 12001)])
def test_library_rows(cuda, dtype, rows, cols):
    x, w, res, _ = inputs(cuda, rows, cols, dtype)
    res = x.flip(0).contiguous()
    y, h = ops.rmsnorm(x, w, 1e-6, residual=res, return_residual=True)
    assert torch.equal(h, x + res)
    hd = h.double()
    close(y, hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-6) * w.double(), dtype)
    close(ops.row_reduce(x, "sum"), x.double().sum(-1), dtype)
    assert torch.equal(ops.row_reduce(x, "amax"), x.amax(-1))
    at = ops.row_reduce(x, "argmin")
    assert bool(((at >= 0) & (at < cols)).all()) and torch.equal(x.gather(-1, at[:, None]), x.amin(-1, keepdim=True))
    assert dtype != torch.float32 or torch.equal(at, x.argmin(-1))  # 16-bit rows have ties
    if cols > 1:
        buf = torch.full(((rows + 2) * cols,), 7.0, dtype=dtype, device=cuda)
        ops.softmax_layernorm(x, w, w, w, 1e-5, out=buf[cols:-cols].view(rows, cols))
        close(buf[cols:-cols].view(rows, cols), chain(*(t.double() for t in (x, w, w, w))), dtype)
        assert bool((buf[:cols] == 7).all()) and bool((buf[-cols:] == 7).all())


def test_products_are_not_rounded_before_they_are_added(cuda):
    """A thread's products meet in one fma, in the vector that the row ends in as in the others:
    -(1 + 2^-11) and (1 + 2^-12)^2 leave 2^-24, which a rounded product would have lost.  Of 64
    threads with five vectors of four, columns 0-3 and 1024-1027 are the first one's, column 4 and
    1028, the last, the second one's."""
    import inductor_x_b200  # noqa: F401
    from torch._inductor.utils import run_and_get_code

    a, b = (torch.zeros(3, 1029, device=cuda) for _ in range(2))
    a[:, :5], b[:, :5] = -(1 + 2.0 ** -11), 1
    a[:, 1024:], b[:, 1024:] = 1 + 2.0 ** -12, 1 + 2.0 ** -12
    torch._dynamo.reset()
    out, code = run_and_get_code(torch.compile(lambda a, b: (a * b).sum(-1), dynamic=False), a, b)
    code = "\n".join(code)
    assert "reduce_dot(" in code and "#define IXB_ROW_TEAM 64" in code and "#define IXB_ROW_VPT 5" in code
    assert torch.equal(out, torch.full_like(out, 5 * 2.0 ** -24))
