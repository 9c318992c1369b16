"""The attention backward's blocks take over pending work items: sizes with more key tiles, or more pairs of
query tiles, than the GPU has SMs, with one and two live query tiles in the last item of a head."""
import math

import pytest
import torch

from inductor_x_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Sq,Sk,causal,dtype", [
    (5, 32, 136, 136, True, torch.bfloat16), (4, 40, 60, 200, True, torch.float16), (2, 33, 640, 640, True, torch.bfloat16),
    (7, 23, 260, 129, False, torch.float16), (2, 40, 500, 1100, False, torch.bfloat16)])
def test_many_items(cuda, B, H, Sq, Sk, causal, dtype):
    g = torch.Generator(device=cuda).manual_seed(Sq + Sk)
    q, dy = (torch.randn(B, H, Sq, 128, generator=g, device=cuda).to(dtype) for _ in range(2))
    k, v = (torch.randn(B, H, Sk, 128, generator=g, device=cuda).to(dtype) for _ in range(2))
    scale = 1 / math.sqrt(128)
    out, lse = ops.fused_attention(q, k, v, scale, causal=causal, return_lse=True)
    got = ops.fused_attention_backward(q, k, v, out, lse, dy, scale, causal=causal, check=True)
    # A few heads alone: a block for each item.  Whoever works on an item, its arithmetic is the same.
    few = [t[-1:, -3:] for t in (q, k, v, out, lse, dy)]
    alone = ops.fused_attention_backward(*few, scale, causal=causal, check=True)
    for a, b in zip(got, alone):
        assert torch.equal(a[-1:, -3:], b)
    # A gradient carries four roundings to 16 bits, each of at most 2^-9 (bf16) or 2^-12 (f16) of a term: the output
    # (in the row sums), the probabilities or their gradients as an operand, and the result; the inputs are exact.
    # In the norm of a head that is at most their sum.  (Single elements have no such bound: a value near zero may
    # be a difference of terms far above the mean.)  A block of rows that is wrong is at least a tenth of the norm.
    bound = 4 * 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    mask = torch.ones(Sq, Sk, dtype=torch.bool, device=cuda).tril(Sk - Sq) if causal else None
    leaves = [t.double().requires_grad_() for t in (q, k, v)]
    ref = torch.nn.functional.scaled_dot_product_attention(*leaves, attn_mask=mask, scale=scale)
    for a, want in zip(got, torch.autograd.grad(ref, leaves, dy.double())):
        error = (a.double() - want).flatten(2).norm(dim=-1) / want.flatten(2).norm(dim=-1)
        assert float(error.max()) <= bound


@pytest.mark.parametrize("B,H,Sq,Sk,causal,dtype", [
    (5, 32, 136, 136, True, torch.bfloat16), (4, 40, 60, 200, True, torch.float16), (7, 23, 260, 129, False, torch.float16)])
def test_many_items_without_scratch(cuda, monkeypatch, B, H, Sq, Sk, causal, dtype):
    """dK/dV blocks that keep no dS and take over items all the same."""
    monkeypatch.setattr(ops, "SCORE_GRADIENT_BYTES", 0)
    test_many_items(cuda, B, H, Sq, Sk, causal, dtype)
