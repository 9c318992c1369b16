"""Lines between the forms of a generated kernel that their sizes decide: which form a group gets on both sides of each.
Emitted for CPU tensors that nothing is read from; one module stands in for all of them, nothing is launched."""
import re

import pytest
import torch

import inductor_x_b200  # noqa: F401
from inductor_x_b200.codegen import jit


@pytest.fixture
def source(dry_backend, monkeypatch):
    from torch._inductor.utils import run_and_get_code

    build, built = jit.compile_source, []

    def one_for_all(src, *args, **kwargs):
        if not built:
            built.append(build(src, *args, **kwargs))
        return built[0]

    monkeypatch.setattr(jit, "compile_source", one_for_all)

    def emitted(fn, *shapes):
        torch._dynamo.reset()
        args = [torch.zeros(n, dtype=torch.int64) if dtype == "index" else torch.empty(n, dtype=dtype) for n, dtype in shapes]
        _, code = run_and_get_code(torch.compile(fn, dynamic=False), *args)
        return "\n".join(code)

    return emitted


F32, F16, BF16 = torch.float32, torch.float16, torch.bfloat16


def test_tiles_with_smaller_ones_at_their_ends(source):
    for shape, dtype, tiled in (((64, 30, 33, 16), F32, False), ((300, 30, 33, 64), F16, False), ((64, 48, 1000, 48), F16, False),
                                ((16, 32, 48, 64), F16, True), ((50, 452, 221, 16), F32, True), ((64, 100, 1300, 64), F16, True)):
        assert ("tile_order<" in source(lambda x: x.permute(0, 2, 1, 3).sum(3), (shape, dtype))) == tiled, shape


def test_rows_that_blocks_are_started_for(source):
    """How many rows' worth of bytes a row moves, which the launch holds against L2; 0 where blocks are resident."""
    for fn, moved in ((lambda x: torch.softmax(x, -1), 2), (lambda x: x.sum(-1), 0)):
        assert f"static constexpr int kStream = {moved};" in source(fn, ((3000, 16), F32))


def test_threads_that_blocks_are_started_from(source):
    def threads(fn, *shapes):
        return int(re.search(r"static constexpr long long kStream = (\d+);", source(fn, *shapes)).group(1))

    n = 1 << 20
    assert 2 ** 24 / 8 < threads(lambda a, b: a + b, ((n,), BF16), ((n,), BF16)) < 2 ** 24.5 / 8    # 100 and 142 MB
    assert threads(lambda a: a.float(), ((n,), BF16)) == 1
    assert threads(lambda a: a * 2, ((n,), BF16)) == threads(lambda a, b: torch.exp(a) * b, ((n,), BF16), ((n,), BF16)) == 0
    assert 2 ** 22 / 16 < threads(lambda x: (x.transpose(1, 2) + 1).contiguous(), ((8, 64, 64), F32)) < 2 ** 23 / 16


@pytest.mark.parametrize("dtype,longer,shorter", [(F16, 333, 127), (F32, 333, 127)])
def test_odd_rows_that_are_picked_or_permuted(source, dtype, longer, shorter):
    for n, walked in ((longer, True), (shorter, False)):
        assert ("launch_pointwise_rows" in source(lambda t, i: t[i], ((301, n), dtype), ((77,), "index"))) == walked
        assert ("launch_pointwise_rows" in source(lambda x: (x.permute(0, 2, 1, 3) * 2).contiguous(), ((2, 5, 6, n), dtype))) == walked


def test_odd_rows_that_share_a_run_or_a_value(source):
    def walked(fn, n, dtype, *others):
        return "launch_pointwise_rows" in source(fn, ((60, n), dtype), *((shape, dtype) for shape in others))

    for n, dtype, one_a_row, shared, part in ((333, F16, False, False, False), (1023, F16, True, False, True), (4097, F16, True, True, True),
                                              (4097, F32, False, False, False)):
        assert walked(lambda x, r: torch.maximum(x, r), n, dtype, (60, 1)) == one_a_row
        assert walked(lambda x, w: torch.maximum(x, w), n, dtype, (n,)) == shared
        assert walked(lambda x: x[:, 2:] * 2, n + 2, dtype) == part
    # arithmetic that a warp with an end in it would do for vectors that are cut
    for n, dtype in ((65, F32), (333, F16), (4097, F16)):
        assert not walked(lambda x, w: torch.nn.functional.gelu(x + w), n, dtype, (n,))


@pytest.mark.parametrize("b,c,dtype,shared", [
    (32, 32, F16, False), (40, 64, F16, False), (40, 96, F16, True), (100, 160, F32, True),      # lanes ordered along the source rows
    (48, 48, F16, False), (72, 48, F16, True), (48, 40, F32, True), (33, 72, F32, False), (127, 72, F32, True),   # rows whole words apart
    (33, 33, F32, False), (129, 129, F16, False), (200, 201, F16, True), (160, 127, F32, True)])
def test_transposes_by_shared_memory(source, b, c, dtype, shared):
    assert ("launch_pointwise_smem" in source(lambda x: (x.transpose(1, 2) + 1).contiguous(), ((3, b, c), dtype))) == shared


def test_digits_by_a_power_of_two_keep_64_bits(source):
    for n, bits in ((4, ""), (8, ""), (12, "32")):
        assert f"idiv{bits}(xindex, {n}LL)" in source(lambda x, r: x * r, ((999, n), F32), ((999, 1), F32))


def test_small_calls(source):
    for shape, shared in (((2, 65, 59), True), ((3, 65, 59), False), ((2, 63, 59), False)):
        assert ("launch_pointwise_smem" in source(lambda x: (x.transpose(1, 2) + 1).contiguous(), (shape, F16))) == shared, shape
    for rows, n, dtype, walked in ((9, 333, F16, True), (13, 333, F16, False), (9, 333, F32, False), (9, 255, F16, False)):
        assert ("launch_pointwise_rows" in source(lambda x, w: torch.maximum(x, w), ((rows, n), dtype), ((n,), dtype))) == walked, (rows, n)
