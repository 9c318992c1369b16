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


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 8])
def test_rows_that_are_no_multiple_of_32_bytes(cuda, offset):
    """Outputs through the C entry: rows on 32-byte boundaries take stores of a whole sector, others of half
    of one; key tiles of which only some columns are cut, masked or past the end."""
    import math

    from inductor_x_b200 import ops
    from inductor_x_b200 import runtime as rt

    B, H, Sq, Sk = 1, 2, 200, 300
    q, k, v = (torch.randn(B, H, s, 128, device=cuda).half() for s in (Sq, Sk, Sk))
    scale = 1 / math.sqrt(128)
    for causal in (False, True):
        want = ops.fused_attention(q, k, v, scale, causal=causal)
        buf = torch.full((B * H * Sq * 136 + 16,), 7.0, dtype=torch.float16, device=cuda)
        out = buf[offset:offset + B * H * Sq * 136].view(B, H, Sq, 136)[..., :128]
        st = rt.load().ixb_fa_fwd(rt.IXB_F16, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None, B, H, Sq, Sk, 128,
                                  *(ops._bhs_strides(t) for t in (q, k, v, out)), scale, int(causal), None, rt.raw_stream(q.device))
        assert st == 0 and torch.equal(out, want)
        mask = torch.ones(Sq, Sk, dtype=torch.bool, device=cuda).tril(Sk - Sq) if causal else None
        ref = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float(), v.float(), attn_mask=mask, scale=scale)
        assert float((want.float() - ref).abs().max()) <= 4e-3
        out.fill_(7)
        assert bool((buf == 7).all())
