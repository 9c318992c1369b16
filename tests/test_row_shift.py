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


def _shape(code):
    return tuple(int(re.search(rf"#define IXB_ROW_{m} (\d+)", code).group(1)) for m in ("TEAM", "VPT", "KREGS")) + \
        tuple(int(re.search(rf"constexpr int {m} = (\d+);", code).group(1)) for m in ("kConsts", "kShiftPeriod"))


@needs_nvcc
@pytest.mark.parametrize("dtype,cols,kind,shape", [
    # nothing is shifted: the shape is that of the length itself
    (torch.float16, 61, "sum", (8, 1, 0, 0, 0)), (torch.bfloat16, 127, "sum", (8, 2, 0, 0, 0)), (torch.float32, 63, "sum", (8, 2, 0, 0, 0)),
    (torch.float16, 511, "scan", (32, 2, 0, 0, 0)), (torch.float16, 511, "pitches", (32, 2, 1, 1, 0)),
    # a row of whole warps whose every place is taken, in the next shape
    (torch.float16, 511, "affine", (32, 3, 2, 2, 8)), (torch.float32, 16379, "affine", (1024, 4, 2, 2, 4)),
    (torch.float32, 16383, "affine", (1024, 5, 2, 2, 4)), (torch.bfloat16, 32767, "affine", (1024, 5, 1, 2, 8)),
    # ... or, where that is more than a thread may hold or its table has no room, in its own
    (torch.float32, 32767, "affine", (1024, 8, 2, 2, 0)), (torch.bfloat16, 65535, "sum", (1024, 8, 0, 0, 0)),
    (torch.bfloat16, 32767, "three", (1024, 4, 2, 3, 0))])
def test_shape_of_odd_rows(dry_backend, dtype, cols, kind, shape):
    x = torch.empty(40, cols + 9).to(dtype)[:, :cols] if kind == "pitches" else torch.empty(40, cols).to(dtype)
    w, b = (torch.empty(cols).to(dtype) for _ in range(2))
    fn, args = {"sum": (lambda x: x.float().sum(-1), (x,)), "scan": (lambda x: x.cumsum(-1), (x,)),
                "pitches": (lambda x, w: (x * w).softmax(-1), (x, w)),
                "affine": (lambda x, w, b: F.layer_norm(x, (cols,), w, b), (x, w, b)),
                "three": (lambda x, w, b, g: F.layer_norm(x, (cols,), w, b) * g, (x, w, b, w + 1))}[kind]
    assert _shape(_period(fn, *args)[2]) == shape


def test_shared_memory_of_every_shape():
    """What the emitter gives a row and what is measured beside it stay within a block's shared memory."""
    from inductor_x_b200.codegen import split_tiling as st

    for dtype, vec in ((torch.float32, 4), (torch.float16, 8)):
        for nvec in sorted({n for k in range(5, 14) for n in (2 ** k - 1, 2 ** k, 2 ** k + 1, 3 * 2 ** k // 2, 5 * 2 ** k // 4)} | {2500}):
            for cols in (nvec * vec, nvec * vec - 1):
                if st.walked_in_chunks(cols, dtype):
                    continue
                base = st.choose_row_config(cols, dtype, rows=1 << 20)
                for n in range(7):
                    cfg = st.covering_config(cols, dtype, base, n, rows=1 << 20)
                    assert cfg is None or cfg is base or st.table_fits(n, st.const_regs(n, cfg.elems_per_thread), cfg.capacity)
                    for team, teams, vpt, _, _, kregs in st.row_candidates(cols, base, n_consts=n, kregs=st.const_regs(n, base.elems_per_thread)):
                        table = max(0, n - kregs) * team * vpt * vec * 4
                        # 32 bytes a warp of exchange, beside 227 KiB a block may have
                        assert team < 32 or table + team * teams <= 227 * 1024


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
@pytest.mark.parametrize("dtype,cols,operands", [(torch.float32, 32767, 2), (torch.float32, 32767, 3), (torch.bfloat16, 32767, 2), (torch.bfloat16, 32767, 3),
                                                 (torch.float16, 65535, 1), (torch.float32, 16383, 5), (torch.bfloat16, 32768, 5)])
def test_long_rows_with_per_column_operands(cuda, dtype, cols, operands):
    """Rows that fill their team, with more per-column operands than registers and shared memory hold."""
    import inductor_x_b200  # noqa: F401

    g = torch.Generator(device=cuda).manual_seed(cols)
    rows = 67
    x = torch.randn(rows, cols, generator=g, device=cuda).to(dtype)
    p = [(1 + 0.1 * torch.randn(cols, generator=g, device=cuda)).to(dtype) for _ in range(operands)]

    def fn(x, *p):
        y = (x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6)) * p[0]
        for n, w in enumerate(p[1:]):
            y = y + w if n % 2 == 0 else y * w
        return y

    torch._dynamo.reset()
    got = torch.compile(lambda x, *p: fn(x.float(), *(w.float() for w in p)).to(dtype), dynamic=False)(x, *p)
    _close(got, fn(x.double(), *(w.double() for w in p)), dtype)


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
