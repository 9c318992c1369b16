"""Forms of a generated kernel that a rule on sizes keeps for large or long operands, on the GPU: at the edges of their tiles,
where the rule would not take them, with the rule set aside; and at sizes that it does take them at."""
import pytest
import torch

import test_odd_rows_gpu as odd_rows
import test_transposes_gpu as transposes
from inductor_x_b200.codegen.kernel import B200Kernel

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_caches():
    """A graph that was compiled under the rule is not taken for one without it."""
    with torch._inductor.config.patch(force_disable_caches=True):
        yield


@pytest.mark.parametrize("dtype,b,c", [(torch.float16, 32, 33), (torch.float16, 58, 121), (torch.float16, 129, 240), (torch.bfloat16, 700, 131),
                                       (torch.float32, 33, 32), (torch.float32, 121, 61), (torch.float32, 65, 120)])
def test_transposes_by_shared_memory(cuda, monkeypatch, no_caches, dtype, b, c):
    from torch._inductor.utils import run_and_get_code

    monkeypatch.setattr(B200Kernel, "_smem_pays", staticmethod(lambda *a: True))
    torch._dynamo.reset()
    x = transposes.data(cuda, (3, b, c), dtype)
    got, code = run_and_get_code(torch.compile(lambda x: (x.transpose(1, 2) + 1.0).contiguous(), dynamic=False), x)
    assert torch.equal(got, x.transpose(1, 2) + 1.0) and "launch_pointwise_smem" in "\n".join(code)


def test_groups_of_transposes_by_shared_memory(cuda, monkeypatch, no_caches):
    monkeypatch.setattr(B200Kernel, "_smem_pays", staticmethod(lambda *a: True))
    transposes.test_groups(cuda)


@pytest.mark.parametrize("dtype,cols", [(torch.float32, 17), (torch.bfloat16, 39), (torch.float16, 15), (torch.bfloat16, 333), (torch.float32, 1023)])
def test_gathered_odd_rows(cuda, monkeypatch, no_caches, dtype, cols):
    monkeypatch.setattr(B200Kernel, "_row_walk_pays", staticmethod(lambda *a: True))
    odd_rows.test_gathered_rows(cuda, dtype, cols)


def test_operands_of_odd_rows(cuda, monkeypatch, no_caches):
    monkeypatch.setattr(B200Kernel, "_row_walk_pays", staticmethod(lambda *a: True))
    odd_rows.test_operands_of_rows(cuda)


def test_a_block_for_every_few_rows(cuda):
    """More rows of one, two and four vectors than stay in L2, whole and ragged ones."""
    for d in (4, 7, 16):
        x = torch.randn((1 << 26) // d + 5, d, generator=torch.Generator(device=cuda).manual_seed(d), device=cuda)
        torch._dynamo.reset()
        got = torch.compile(lambda x: torch.softmax(x, -1), dynamic=False)(x)
        assert float((got - torch.softmax(x, -1)).abs().max()) <= 1e-6


def test_a_block_for_256_vectors(cuda):
    for n in (1 << 25, (1 << 25) + 9):
        a, b = (torch.randn(n, generator=torch.Generator(device=cuda).manual_seed(i), device=cuda).to(torch.bfloat16) for i in range(2))
        torch._dynamo.reset()
        assert torch.equal(torch.compile(lambda a, b: a + b, dynamic=False)(a, b), a + b)
