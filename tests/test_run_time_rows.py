"""Row lengths that are sizes of the call (``dynamic=True``): a module serves every row up to the
capacity of the shape compiled for the first length seen, which is the power-of-two cover of that
length - a shape cut to fit it would refuse the next longer row."""
import re

import pytest
import torch

# first length seen and the capacity of its power-of-two cover
LENGTHS = [(torch.float32, 384, 512), (torch.float32, 600, 1024), (torch.float32, 3072, 4096), (torch.bfloat16, 1100, 2048),
           (torch.bfloat16, 4100, 8192)]


@pytest.mark.parametrize("dtype,first,capacity", LENGTHS)
def test_shape_of_a_run_time_length_is_not_cut_to_fit(dry_backend, dtype, first, capacity):
    from torch._inductor.utils import run_and_get_code

    torch._dynamo.reset()
    _, code = run_and_get_code(torch.compile(lambda t: torch.softmax(t, -1), dynamic=True), torch.randn(33, first).to(dtype))
    code = "\n".join(code)
    team, vpt = (int(re.search(rf"#define IXB_ROW_{m} (\d+)", code).group(1)) for m in ("TEAM", "VPT"))
    assert "constexpr int kCols = 0;" in code
    assert team * vpt * (16 // dtype.itemsize) == capacity


def test_graph_cache_tells_run_time_lengths_apart():
    """The key of a compiled graph holds the power-of-two class of each run-time size."""
    from torch._guards import TracingContext, tracing
    from torch._subclasses import FakeTensorMode
    from torch.fx.experimental.symbolic_shapes import DimDynamic, ShapeEnv, StatelessSymbolicContext

    from inductor_x_b200.fusion_attention_graph import B200AttentionPass

    def key(rows, cols):
        mode = FakeTensorMode(shape_env=ShapeEnv())
        mode.from_tensor(torch.empty(rows, cols), symbolic_context=StatelessSymbolicContext([DimDynamic.DYNAMIC] * 2))
        with tracing(TracingContext(mode)):
            return B200AttentionPass().uuid()

    assert key(33, 384) == key(40, 512) == key(64, 257)
    assert len({key(33, 384), key(33, 600), key(33, 256), key(384, 33), B200AttentionPass().uuid()}) == 5


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,first,capacity", LENGTHS)
def test_lengths_up_to_the_capacity(cuda, dtype, first, capacity):
    import inductor_x_b200  # noqa: F401

    torch._dynamo.reset()
    fn = torch.compile(lambda t: torch.softmax(t, -1), dynamic=True)
    g = torch.Generator().manual_seed(first)
    tol = {torch.float32: 1e-5, torch.bfloat16: 8e-3}[dtype]  # 32-bit sums, one rounding of the result
    # (Inductor's graph cache is on: it must not bring the module of another case's first length)
    for cols in (first, first + 1, first - 1, capacity - 1, capacity):
        x = torch.randn(33, cols, generator=g).to(dtype).to(cuda)
        torch.testing.assert_close(fn(x).double(), torch.softmax(x.double(), -1), rtol=tol, atol=1e-6)
