"""Sums over the rows emitted inside the row kernel that works on the same rows (the gradient of a norm's
weight beside that of its input)."""
import re
import shutil

import pytest
import torch

from inductor_x_b200 import config

needs_nvcc = pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")


def _norm(x, w):
    return (x.float() * torch.rsqrt(x.float().square().mean(-1, keepdim=True) + 1e-6) * w.float()).to(x.dtype)


def _dx_dw(x, w, dy, rstd):
    """What a norm's backward does, with the sum over the rows first."""
    h = dy.float() * w.float()
    dw = (dy.float() * x.float() * rstd).sum(0)
    dx = (h * rstd - x.float() * (h * x.float()).mean(-1, keepdim=True) * rstd ** 3).to(x.dtype)
    return dw, dx


def _code(fn, *args):
    from torch._inductor.utils import run_and_get_code

    torch._dynamo.reset()
    return "\n".join(run_and_get_code(torch.compile(fn, dynamic=False), *args)[1])


@needs_nvcc
def test_both_gradients_come_from_one_kernel(dry_backend):
    x, dy = (torch.randn(4096, 4096).bfloat16() for _ in range(2))
    w, rstd = torch.randn(4096).bfloat16(), torch.rand(4096, 1)
    code = _code(_dx_dw, x, w, dy, rstd)
    assert code.count("ixb_load_kernel('''") == 1 and code.count("kColumns = 1;") == 1
    assert code.count("finish_columns<float>") == 1 and re.search(r"del ixb_partials_\d+", code)


@needs_nvcc
def test_sums_behind_the_row_kernel_and_their_conversions(dry_backend):
    """A layer norm's backward: two sums behind the row kernel in the graph, converted to the type of the
    weights."""
    import torch.nn.functional as F
    from torch._inductor.utils import run_and_get_code

    leaves = [t.requires_grad_(True) for t in (torch.randn(4096, 4096).bfloat16(), *(torch.randn(4096).bfloat16() for _ in range(2)))]

    def step(*leaves):
        y = torch.compile(lambda x, w, b: F.layer_norm(x, (4096,), w, b), dynamic=False)(*leaves)
        return torch.autograd.grad(y, leaves, torch.ones_like(y))

    torch._dynamo.reset()
    code = run_and_get_code(step, *leaves)[1][-1]
    assert code.count("ixb_load_kernel('''") == 1 and code.count("kColumns = 2;") == 1
    assert code.count("finish_columns<ixb::bf16>") == 2


@needs_nvcc
@pytest.mark.parametrize("why", ["off", "few rows", "small", "wide", "other order", "used between", "short rows"])
def test_what_stays_a_kernel_of_its_own(dry_backend, monkeypatch, why):
    rows, cols = {"few rows": (100, 65536), "small": (1024, 4096), "wide": (2048, 32768 * 4), "short rows": (1 << 18, 128)}.get(why, (4096, 4096))
    monkeypatch.setattr(config, "merged_column_sums", why != "off")
    x, dy = (torch.empty(rows, cols, dtype=torch.bfloat16) for _ in range(2))
    w, rstd = torch.empty(cols, dtype=torch.bfloat16), torch.empty(rows, 1)
    fn = _dx_dw
    if why == "other order":
        x = torch.empty(cols, rows, dtype=torch.bfloat16).t()
    if why == "used between":         # the row kernel wants the sum
        def fn(x, w, dy, rstd):
            dw, _ = _dx_dw(x, w, dy, rstd)
            return dw, (x.float() * dw).softmax(-1)
    code = _code(fn, x, w, dy, rstd)
    assert not re.search(r"kColumns = [1-9]", code) and "ixb_partials" not in code


@needs_nvcc
@pytest.mark.parametrize("cols,into", [(32769, torch.float32), (40960, torch.float32), (40960, torch.bfloat16), (65536, torch.float32)])
def test_rows_walked_in_chunks_leave_the_sums_to_a_kernel_of_their_own(dry_backend, cols, into):
    """fp32 rows of more than 8192 vectors; a sum that is converted to 16 bits does not make them shorter."""
    x, dy = (torch.empty(256, cols) for _ in range(2))
    w, rstd = torch.empty(cols), torch.empty(256, 1)

    def fn(x, w, dy, rstd):
        dw, dx = _dx_dw(x, w, dy, rstd)
        return dw.to(into), dx

    code = _code(fn, x, w, dy, rstd)
    assert code.count("kLooped = true;") == 1 and code.count("ixb_load_kernel('''") >= 2
    assert not re.search(r"kColumns = [1-9]", code) and "ixb_partials" not in code


@pytest.mark.parametrize("dtype,rows,cols,sums,pays", [
    # one sum over whole vectors beside a team of 1024 threads
    (torch.bfloat16, 4096, 16384, 1, False), (torch.bfloat16, 1024, 24576, 1, False), (torch.float32, 4096, 16384, 1, True),
    (torch.float32, 1024, 24576, 1, False), (torch.float32, 256, 16384, 1, False), (torch.float32, 400, 8192, 1, True),
    # beside fewer threads
    (torch.bfloat16, 1024, 12288, 1, True), (torch.bfloat16, 400, 8192, 1, True), (torch.bfloat16, 256, 12288, 1, False),
    # rows of other lengths
    (torch.bfloat16, 220, 16000, 1, True), (torch.bfloat16, 200, 16383, 1, True), (torch.bfloat16, 1024, 24571, 1, True),
    (torch.bfloat16, 512, 32767, 1, False), (torch.bfloat16, 2048, 32767, 1, True), (torch.bfloat16, 150, 32767, 1, False),
    (torch.float32, 256, 16383, 1, True), (torch.float32, 256, 32767, 1, False), (torch.bfloat16, 300, 50257, 1, False),
    (torch.bfloat16, 512, 65535, 1, False), (torch.bfloat16, 512, 65529, 1, False),
    # two sums
    (torch.bfloat16, 400, 16384, 2, True), (torch.bfloat16, 256, 16384, 2, False), (torch.bfloat16, 1024, 32768, 2, True),
    (torch.bfloat16, 512, 32767, 2, False), (torch.float32, 1024, 20000, 2, True), (torch.float32, 512, 16383, 2, True),
    (torch.float32, 512, 32767, 2, False), (torch.bfloat16, 2048, 32767, 2, False)])
def test_where_one_kernel_is_quicker(dtype, rows, cols, sums, pays):
    from inductor_x_b200.codegen import scheduling, split_tiling

    group = scheduling.ColumnGroup([], [], [], set(), rows, cols)
    group.sums = [None] * sums
    shape = split_tiling.choose_row_config(cols, dtype, rows=rows)
    assert group._pays(shape, dtype) == pays
    # whatever pays leaves a thread of the shape in use no more sums than it has registers
    used = shape if cols % shape.vec == 0 else split_tiling.covering_config(cols, dtype, shape, 0, rows=rows) or shape
    assert not pays or used.elems_per_thread * sums <= 65536 // (used.team * used.teams)


@needs_nvcc
@pytest.mark.parametrize("dtype,rows,cols", [(torch.bfloat16, 300, 65535), (torch.bfloat16, 1024, 16384), (torch.float32, 300, 32768)])
def test_long_rows_keep_their_registers(dry_backend, dtype, rows, cols):
    x, dy = (torch.empty(rows, cols, dtype=dtype) for _ in range(2))
    code = _code(_dx_dw, x, torch.empty(cols, dtype=dtype), dy, torch.empty(rows, 1))
    assert not re.search(r"kColumns = [1-9]", code) and "ixb_partials" not in code


@needs_nvcc
@pytest.mark.parametrize("rows,partials", [(413, 416), (4096, 592)])
def test_partial_sums_are_as_many_as_blocks(dry_backend, rows, partials):
    """No more rows of partial sums than there are blocks: one for each row, rounded up to whole periods of
    the offsets from a boundary, or four an SM."""
    cols = 8003
    x, dy = (torch.empty(rows, cols, dtype=torch.bfloat16) for _ in range(2))
    code = _code(_dx_dw, x, torch.empty(cols, dtype=torch.bfloat16), dy, torch.empty(rows, 1))
    assert "kShiftPeriod = 8;" in code and f"kPartials = {partials};" in code
    assert re.search(rf"ixb_partials_\d+ = empty_strided_cpu\(\({partials * 8004},\)", code)


TOL = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def _close(got, want, dtype):
    assert got.dtype == dtype
    err = (got.double() - want).abs() / want.abs().clamp_min(float(want.square().mean().sqrt()))
    assert float(err.max()) <= TOL[dtype]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,rows,cols", [
    (torch.bfloat16, 2048, 4096), (torch.float32, 1500, 4096), (torch.float16, 5003, 1537), (torch.float32, 1031, 4097),
    (torch.bfloat16, 1025, 8191), (torch.float16, 20000, 264), (torch.bfloat16, 9000, 520), (torch.float16, 1024, 16384),
    (torch.bfloat16, 131, 8193), (torch.float32, 401, 8192)])
def test_training_step_of_a_norm(cuda, monkeypatch, dtype, rows, cols):
    """Rows that are no whole number of blocks, several teams a block, odd rows (whose blocks keep to one
    offset), one team of many warps; against 64 bits.  The sum's bound: fp32 partial sums of `rows` terms,
    rounded once."""
    import inductor_x_b200  # noqa: F401
    from inductor_x_b200.codegen import jit

    monkeypatch.setattr(config, "column_sum_elements", 1 << 20)
    monkeypatch.setattr(config, "column_sum_elements_odd", 1 << 20)
    g = torch.Generator(device=cuda).manual_seed(rows)
    x, dy = (torch.randn(rows, cols, generator=g, device=cuda).to(dtype) for _ in range(2))
    w = (1 + 0.1 * torch.randn(cols, generator=g, device=cuda)).to(dtype)
    a, b = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    torch._dynamo.reset()
    y = torch.compile(_norm, dynamic=False)(a, b)
    for _ in range(2):               # the second time in the launch shape that measured fastest
        dx, dw = torch.autograd.grad(y, (a, b), dy, retain_graph=True)
    assert any("kColumns = 1;" in k.src and f"partial_pitch({cols})" in k.src for k in jit._loaded.values())
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    yd = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * wd
    ex, ew = torch.autograd.grad(yd, (xd, wd), dy.double())
    _close(y.detach(), yd.detach(), dtype)
    _close(dx, ex, dtype)
    _close(dw, ew, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(256, 32769), (203, 50257)])
def test_training_step_of_rows_walked_in_chunks(cuda, rows, cols):
    """fp32 rows longer than a block holds, of a size whose sums would otherwise come out of the row kernel."""
    import inductor_x_b200  # noqa: F401

    g = torch.Generator(device=cuda).manual_seed(rows)
    x, dy = (torch.randn(rows, cols, generator=g, device=cuda) for _ in range(2))
    w = 1 + 0.1 * torch.randn(cols, generator=g, device=cuda)
    a, b = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    torch._dynamo.reset()
    dx, dw = torch.autograd.grad(torch.compile(_norm, dynamic=False)(a, b), (a, b), dy)
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    yd = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * wd
    ex, ew = torch.autograd.grad(yd, (xd, wd), dy.double())
    _close(dx, ex, torch.float32)
    _close(dw, ew, torch.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(3000, 1024), (1500, 3001)])
def test_training_step_of_a_layer_norm(cuda, monkeypatch, rows, cols):
    import torch.nn.functional as F

    import inductor_x_b200  # noqa: F401

    monkeypatch.setattr(config, "column_sum_elements", 1 << 20)
    monkeypatch.setattr(config, "column_sum_elements_odd", 1 << 20)
    g = torch.Generator(device=cuda).manual_seed(rows)
    x, dy = (torch.randn(rows, cols, generator=g, device=cuda).half() for _ in range(2))
    w, b = ((1 + 0.1 * torch.randn(cols, generator=g, device=cuda)).half() for _ in range(2))
    leaves = [t.clone().requires_grad_(True) for t in (x, w, b)]
    torch._dynamo.reset()
    y = torch.compile(lambda x, w, b: F.layer_norm(x, (cols,), w, b), dynamic=False)(*leaves)
    got = torch.autograd.grad(y, leaves, dy)
    wide = [t.double().requires_grad_(True) for t in (x, w, b)]
    want = torch.autograd.grad(F.layer_norm(wide[0], (cols,), wide[1], wide[2]), wide, dy.double())
    for a, e in zip(got, want):
        _close(a, e, torch.float16)


@pytest.mark.gpu
def test_sums_whose_operand_is_overwritten(cuda):
    """The row kernel may write its result over an operand that the sum reads as well; NaN in one column
    stays there."""
    import inductor_x_b200  # noqa: F401

    g = torch.Generator(device=cuda).manual_seed(1)
    rows, cols = 3001, 2053

    def fn(x, dy, rstd):
        t = dy * 2 + 1                       # a buffer of the graph's own, free to be written over
        t = torch.ops.aten.cumsum(t, 0)      # (an extern kernel keeps it from being computed twice)
        s = (t * x * rstd).sum(0)
        return s, t * rstd - x * (t * x).mean(-1, keepdim=True)

    x, dy = (torch.randn(rows, cols, generator=g, device=cuda) for _ in range(2))
    dy = dy * 1e-2 - 0.5
    rstd = torch.rand(rows, 1, generator=g, device=cuda)
    x[7, 5] = float("nan")
    torch._dynamo.reset()
    s, d = torch.compile(fn, dynamic=False)(x, dy, rstd)
    es, ed = fn(x.double(), dy.double(), rstd.double())
    assert bool(s[5].isnan()) and int(s.isnan().sum()) == 1 and int(d.isnan().any(1).sum()) == 1
    keep = torch.arange(cols, device=cuda) != 5
    # (the cumulated operand is itself a sum of up to 3001 fp32 terms)
    assert float((s.double() - es)[keep].abs().max() / es[keep].abs().max()) <= 1e-4
    live = torch.arange(rows, device=cuda) != 7
    assert float((d.double() - ed)[live].abs().max() / ed[live].abs().max()) <= 1e-4


@pytest.mark.gpu
def test_bandwidth_print_counts_the_operands(cuda, capsys, monkeypatch):
    """config.profile_bandwidth: three matrices and three vectors, without the workspace of partial sums."""
    import inductor_x_b200  # noqa: F401

    rows = cols = 4096
    x, dy = (torch.randn(rows, cols, device=cuda).bfloat16() for _ in range(2))
    w, rstd = torch.randn(cols, device=cuda).bfloat16(), torch.rand(rows, 1, device=cuda)
    torch._dynamo.reset()
    fn = torch.compile(_dx_dw, dynamic=False)
    fn(x, w, dy, rstd)
    capsys.readouterr()
    monkeypatch.setattr(config, "profile_bandwidth", True)
    fn(x, w, dy, rstd)
    lines = re.findall(r"ms\s+([\d.]+)GB", capsys.readouterr().out)
    assert len(lines) == 1 and abs(float(lines[0]) - (3 * 2 * rows * cols + 2 * cols + 4 * rows + 4 * cols) / 1e9) <= 1e-3
