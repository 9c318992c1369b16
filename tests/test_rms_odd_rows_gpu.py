"""RMSNorm of rows off a 16-byte boundary: every launch shape of the kernel that works in the vectors of
memory, bases that share an offset and bases that do not (the general kernel), rows in place.  Against
64-bit arithmetic; results are 32-bit sums rounded once."""
import pytest
import torch

from inductor_x_b200 import runtime as rt

pytestmark = pytest.mark.gpu
TOL = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}


def guarded(t, offset):
    """A copy of t `offset` elements behind a 16-byte boundary, between sentinels."""
    buf = torch.full((t.numel() + 64,), 7.0, dtype=t.dtype, device=t.device)
    view = buf[16 + offset:16 + offset + t.numel()].view(t.shape)
    view.copy_(t)
    return buf, view


def check(rows, cols, dtype, residual, offsets, in_place=False):
    g = torch.Generator(device="cuda").manual_seed(rows * 40009 + cols)
    x, res = (torch.randn(rows, cols, generator=g, device="cuda").to(dtype) for _ in range(2))
    w = (1 + 0.1 * torch.randn(cols, generator=g, device="cuda")).to(dtype)
    h = x + res if residual else x
    hd = h.double()
    want = hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    (bx, vx), (br, vr), (bw, vw) = guarded(x, offsets[0]), guarded(res, offsets[1]), guarded(w, offsets[2])
    (by, vy), (bh, vh) = guarded(torch.zeros_like(x), offsets[3]), guarded(torch.zeros_like(x), offsets[4])
    if in_place:
        by, vy = bx, vx
    rt.check("ixb_rmsnorm", rt.load().ixb_rmsnorm(
        rt.DTYPE_CODE[dtype], vx.data_ptr(), vr.data_ptr() if residual else None, vw.data_ptr(), vy.data_ptr(),
        vh.data_ptr() if residual else None, rows, cols, 1e-6, None, rt.raw_stream(x.device)))
    err = (vy.double() - want).abs() / want.abs().clamp_min(float(want.square().mean().sqrt()))
    assert float(err.max()) <= TOL[dtype]
    if residual:
        assert torch.equal(vh, h)
        vh.zero_()
        assert bool((bh[:16 + offsets[4]] == 7).all()) and bool((bh[16 + offsets[4] + x.numel():] == 7).all())
    assert bool((by[:16 + offsets[3]] == 7).all()) and bool((by[16 + offsets[3] + x.numel():] == 7).all())


# lengths around the capacities of the launch shapes (in vectors 32, 64, 96, 128, 192, ... 4096: a row may
# touch one vector more than its length fills), one element, rows with fewer of one offset than blocks
VECTORS = [32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("residual", [False, True])
def test_launch_shapes(cuda, dtype, residual):
    vec = 16 // torch.empty(0, dtype=dtype).element_size()
    for n in VECTORS:
        for cols in (n * vec - 2 * vec + 1, n * vec - 1):
            check(11, cols, dtype, residual, (0, 0, 0, 0, 0))
    for rows, cols in ((1, 1), (1000, 1), (700, 7), (2000, 41), (1, 515), (9, 1538), (13, 2052)):
        check(rows, cols, dtype, residual, (0, 0, 0, 0, 0))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("cols", [64, 333, 1026])
def test_bases_off_a_boundary(cuda, dtype, cols):
    vec = 16 // torch.empty(0, dtype=dtype).element_size()
    for offset in (1, vec // 2, vec - 1):
        check(37, cols, dtype, True, (offset,) * 5)
        check(37, cols, dtype, True, (offset, offset, 0, offset, offset))
        check(37, cols, dtype, True, (offset, 0, 1, offset, offset))   # no common offset: the general kernel
        check(37, cols, dtype, True, (0, 0, 0, offset, 0))
        check(37, cols, dtype, False, (offset,) * 5, in_place=True)
    check(37, cols, dtype, True, (0,) * 5, in_place=True)
