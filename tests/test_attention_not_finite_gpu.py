"""NaN and infinities in the attention forward, where keys are shared over clusters of 1, 2, 4 and 8 blocks and
where they are not: rows that are not finite in 64-bit arithmetic, and only those, are not finite in the result."""
import math

import pytest
import torch

from inductor_x_b200 import ops

pytestmark = pytest.mark.gpu
SCALE = 1 / math.sqrt(128)


def inputs(b, h, sq, sk):
    g = torch.Generator(device="cuda").manual_seed(sq * 8191 + sk)
    return [torch.randn(b, h, s, 128, generator=g, device="cuda").to(torch.bfloat16) for s in (sq, sk, sk)]


def reference(q, k, v, causal):
    s = q.double() @ k.double().transpose(-1, -2) * SCALE
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[-2:], dtype=torch.bool, device="cuda").tril(s.shape[-1] - s.shape[-2]), -math.inf)
    return torch.softmax(s, -1) @ v.double(), torch.logsumexp(s, -1)


# query tiles of one row, of a part, whole ones and several; heads and keys that give clusters of 8 down to none
@pytest.mark.parametrize("b,h,sq,sk", [(1, 2, 1, 2879), (1, 2, 200, 1300), (1, 16, 3, 2500), (2, 4, 300, 700), (2, 16, 3, 300),
                                       (2, 8, 400, 2500), (3, 32, 100, 1300), (2, 16, 400, 700), (5, 32, 300, 700)])
@pytest.mark.parametrize("causal", [False, True])
def test_not_finite(cuda, b, h, sq, sk, causal):
    q, k, v = inputs(b, h, sq, sk)
    whole = ops.fused_attention(q, k, v, SCALE, causal=causal, return_lse=True)

    def check(what, q, k, v, fine=whole):
        got = ops.fused_attention(q, k, v, SCALE, causal=causal, return_lse=True)
        for a, want, was in zip(got, reference(q, k, v, causal), fine):
            finite = torch.isfinite(want)
            assert torch.equal(torch.isfinite(a), finite), what
            assert torch.equal(a[finite], was[finite]), what   # and what is finite is what it was
        assert bool(got[1][~torch.isfinite(got[1])].isnan().all()), what   # whichever kernel it was

    def with_one(t, value, *place):
        t = t.clone()
        t[place] = value
        return t

    check("NaN in a query", with_one(q, math.nan, 0, -1, sq // 2, 5), k, v)
    # (every row sees the first key; the softmax of a score of +inf is NaN)
    plus = with_one(k, 1.0, 0, -1, 0, 5)
    check("+inf in a query", with_one(q, math.inf, 0, -1, sq // 2, 5), plus, v,
          ops.fused_attention(q, plus, v, SCALE, causal=causal, return_lse=True))
    # (under the mask the first half of the rows does not see this key)
    check("NaN in a key", q, with_one(k, math.nan, 0, 0, sk - sq // 2 - 1, 7), v)
    check("NaN in a value", q, k, with_one(v, math.nan, 0, 0, 0, 9))
    check("-inf in a value", q, k, with_one(v, -math.inf, 0, 0, 0, 9))
