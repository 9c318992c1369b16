"""The fused-attention forward takes several work items per thread block: sizes that give fewer
items than the GPU has SMs, a few more, and many more, with one and two live query tiles in the
last item of a head.  Against attention in 32 bits on the same inputs; 2e-2 of max(|expected|,
rms of the row), as for the other attention tests: the probabilities are 16-bit operands."""
import math

import pytest
import torch

from inductor_x_b200 import ops
from oracle import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,causal", [(torch.bfloat16, True), (torch.float16, False)])
@pytest.mark.parametrize("B,H,Sq,Sk", [(1, 37, 1, 129), (3, 50, 200, 200), (5, 32, 300, 300), (2, 33, 1100, 1100),
                                       (7, 31, 129, 385)])
def test_many_items(cuda, dtype, causal, B, H, Sq, Sk):
    g = torch.Generator(device=cuda).manual_seed(B * Sq + Sk)
    q = torch.randn(B, H, Sq, 128, generator=g, device=cuda).to(dtype)
    k, v = (torch.randn(B, H, Sk, 128, generator=g, device=cuda).to(dtype) for _ in range(2))
    scale = 1 / math.sqrt(128)
    out, lse = ops.fused_attention(q, k, v, scale, causal=causal, return_lse=True, check=True)
    s = torch.matmul(q.float(), k.float().transpose(-1, -2)) * scale
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Sk, dtype=torch.bool, device=cuda).tril(Sk - Sq), -math.inf)
    want = torch.matmul(torch.softmax(s, -1), v.float())
    assert graphs.max_rel_err(out, want, dim=-1) <= 2e-2
    assert float((lse - torch.logsumexp(s, -1)).abs().max()) <= 2e-3
    again = ops.fused_attention(q, k, v, scale, causal=causal)
    assert torch.equal(out, again)  # whoever works on an item, its arithmetic is the same
