"""Attention forward whose keys are shared by the slots of a block and the blocks of a cluster: few query rows,
few heads.  Against 64-bit arithmetic on the same inputs; P is rounded to 16 bits before its product."""
import math

import pytest
import torch

from inductor_x_b200 import ops
from tests.test_attention_plan import plan

pytestmark = pytest.mark.gpu


def check(b, h, sq, sk, causal, dtype=torch.bfloat16, bsnd=False):
    g = torch.Generator(device="cuda").manual_seed(sq * 8191 + sk)

    def heads(s):
        if bsnd:
            return torch.randn(b, s, h, 128, generator=g, device="cuda").to(dtype).transpose(1, 2)
        return torch.randn(b, h, s, 128, generator=g, device="cuda").to(dtype)

    q, k, v = heads(sq), heads(sk), heads(sk)
    out, lse = ops.fused_attention(q, k, v, 1 / math.sqrt(128), causal=causal, return_lse=True)
    s = q.double() @ k.double().transpose(-1, -2) / math.sqrt(128)
    if causal:
        s = s.masked_fill(~torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril(sk - sq), -math.inf)
    want = torch.softmax(s, -1) @ v.double()
    rms = want.square().mean().sqrt()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert float((out.double() - want).norm() / want.norm()) <= 1.5 * eps
    assert float(((out.double() - want).abs() / want.abs().clamp_min(float(rms))).max()) <= 12 * eps
    assert float((lse.double() - torch.logsumexp(s, -1)).abs().max()) <= 2e-5
    assert torch.equal(out, ops.fused_attention(q, k, v, 1 / math.sqrt(128), causal=causal))  # one order of adding


# one head to many (clusters of eight blocks down to one), rows of one tile and its edges, key tiles that the
# slots share evenly, unevenly, and fewer of them than slots
FEW_ROWS_HEADS = [(1, 1), (1, 4), (1, 16), (2, 20), (7, 16), (13, 16)]
FEW_ROWS = [(1, 129), (1, 2879), (5, 257), (127, 1024), (128, 1153), (64, 2049)]
FEW_HEADS = [(129, 129), (300, 1000), (512, 512), (1000, 1000), (640, 3000)]


def test_every_cluster_size_is_among_these(cuda):
    """On a B200; what is 0 here runs in fa_fwd_kernel."""
    rows = {plan(b, h, sq, sk)[1] for b, h in FEW_ROWS_HEADS for sq, sk in FEW_ROWS}
    heads = {plan(1, h, sq, sk)[1] for h in (1, 3, 8) for sq, sk in FEW_HEADS}
    assert rows == {0, 1, 2, 4, 8} and heads == {0, 2, 4, 8}
    assert plan(2, 16, 400, 700)[1] == 1     # several query tiles, a block each (test_empty_slots_and_hidden_keys)


@pytest.mark.parametrize("b,h", FEW_ROWS_HEADS)
@pytest.mark.parametrize("sq,sk", FEW_ROWS)
def test_few_rows(cuda, b, h, sq, sk):
    for causal in (False, True):
        check(b, h, sq, sk, causal)


@pytest.mark.parametrize("sq,sk", FEW_HEADS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_few_heads(cuda, sq, sk, dtype):
    for h, causal in ((1, True), (3, False), (8, True)):
        check(1, h, sq, sk, causal, dtype, bsnd=causal)


def test_empty_slots_and_hidden_keys(cuda):
    """Under a causal mask with as many keys as queries the first query tile sees one key tile, so all slots
    but one are empty; rows whose keys lie in the first of several tiles have slots that see nothing."""
    check(1, 2, 1024, 1024, True)
    check(1, 1, 130, 2000, True)
    check(2, 2, 3, 128 * 17 + 1, True)
    check(2, 16, 400, 700, True)
