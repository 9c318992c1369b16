"""The attention backward with dS kept in scratch (ixb_fa_bwd_scratch)."""
import math
import os
import subprocess
import sys

import pytest
import torch

from inductor_x_b200 import ops
from inductor_x_b200 import runtime as rt
from oracle import graphs

TILE = 128 * 128 * 2


def _tiles(Sq, Sk, causal):
    """Tiles of 128 keys x 128 queries in which some query sees some key."""
    return sum(not causal or kv <= q + 127 + (Sk - Sq) for kv in range(0, Sk, 128) for q in range(0, Sq, 128))


@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("Sq,Sk", [(1, 1), (128, 128), (129, 129), (1000, 1000), (130, 450), (1, 4096), (200, 263), (384, 640)])
def test_scratch_size(Sq, Sk, causal):
    per_head = _tiles(Sq, Sk, causal) * TILE
    size = lambda heads, limit: rt.load().ixb_fa_bwd_scratch_bytes(1, heads, Sq, Sk, causal, limit)
    assert size(3, 1 << 40) == 3 * per_head
    assert size(3, 3 * per_head - 1) == 2 * per_head       # two launches of two heads and one
    assert size(7, 4 * per_head) == 4 * per_head
    assert size(9, 4 * per_head) == 3 * per_head           # three equal launches instead of 4 + 4 + 1
    assert size(3, per_head - 1) == 0 and size(0, 1 << 40) == 0


def test_scratch_arguments():
    assert rt.load().ixb_fa_bwd_scratch_bytes(1, 1, 256, 128, 1, 1 << 40) == 0   # refused by the kernels as well
    assert rt.load().ixb_fa_bwd_scratch_bytes(-1, 1, 128, 128, 0, 1 << 40) == 0


# Tolerance as for the backward without scratch: probabilities and their gradients are 16-bit operands.
TOL = {torch.bfloat16: 4e-2, torch.float16: 8e-3}


@pytest.mark.gpu
@pytest.mark.parametrize("Sq,Sk,causal,dtype", [
    (128, 128, True, torch.bfloat16), (129, 129, True, torch.float16), (77, 77, False, torch.float16), (640, 640, True, torch.float16),
    (130, 450, True, torch.float16), (257, 384, True, torch.bfloat16), (300, 130, False, torch.float16), (1, 300, True, torch.float16)])
def test_backward_with_room_for_some_heads(cuda, monkeypatch, Sq, Sk, causal, dtype):
    """Odd numbers of query tiles, ragged ends of both lengths, tiles past the diagonal; five heads in one
    launch, in two of three and two (the scratch holds three), and without room for one."""
    g = torch.Generator().manual_seed(Sq + Sk)
    q, dy = (torch.randn(1, 5, Sq, 128, generator=g).to(dtype) for _ in range(2))
    k, v = (torch.randn(1, 5, Sk, 128, generator=g).to(dtype) for _ in range(2))
    scale = 1 / math.sqrt(128)
    want = graphs.attention_backward(q, k, v, dy, scale, causal=causal)
    qd, kd, vd, dyd = (t.to(cuda) for t in (q, k, v, dy))
    out, lse = ops.fused_attention(qd, kd, vd, scale, causal=causal, return_lse=True, check=True)
    per_head = _tiles(Sq, Sk, causal) * TILE
    for room in (5 * per_head, 3 * per_head, per_head - 1):
        monkeypatch.setattr(ops, "SCORE_GRADIENT_BYTES", room)
        got = ops.fused_attention_backward(qd, kd, vd, out, lse, dyd, scale, causal=causal, check=True)
        for name, a, e in zip(("dq", "dk", "dv"), got, want):
            assert graphs.max_rel_err(a.float().cpu(), e) <= TOL[dtype], (name, room)


@pytest.mark.gpu
def test_keys_past_the_end_do_not_reach_dq(cuda, monkeypatch):
    """All scores far below zero: exp(0 - lse), what the zeros past the last key would give, overflows.
    Both ways round dS to 16 bits before the same product, so they are as close as its roundings."""
    g = torch.Generator().manual_seed(9)
    q, dy = (torch.randn(1, 2, 130, 128, generator=g).to(torch.bfloat16).to(cuda) for _ in range(2))
    k, v = (torch.randn(1, 2, 130, 128, generator=g).to(torch.bfloat16).to(cuda) for _ in range(2))
    q, k = q + 3.25, k - 3.25
    scale = 1 / math.sqrt(128)
    out, lse = ops.fused_attention(q, k, v, scale, return_lse=True, check=True)
    assert float(lse.max()) < -89                              # exp(89) is past the largest float
    got = ops.fused_attention_backward(q, k, v, out, lse, dy, scale, check=True)
    monkeypatch.setattr(ops, "SCORE_GRADIENT_BYTES", 0)
    want = ops.fused_attention_backward(q, k, v, out, lse, dy, scale, check=True)
    for a, e in zip(got, want):
        assert bool(a.isfinite().all()) and graphs.max_rel_err(a.float().cpu(), e.float().cpu()) <= TOL[torch.bfloat16]


@pytest.mark.gpu
def test_scratch_must_be_aligned(cuda):
    q = torch.zeros(1, 1, 8, 128, dtype=torch.bfloat16, device=cuda)
    st = ops._bhs_strides(q)
    f = torch.zeros(64, device=cuda)
    scratch = torch.zeros(2 * TILE, dtype=torch.uint8, device=cuda)
    assert rt.load().ixb_fa_bwd_scratch(rt.IXB_BF16, *[q.data_ptr()] * 5, f.data_ptr(), *[q.data_ptr()] * 3, f.data_ptr(),
                                        scratch.data_ptr() + 8, TILE, 1, 1, 8, 8, 128, *[st] * 8, 1.0, 0, None,
                                        rt.raw_stream(q.device)) == rt.IXB_ERR_ALIGN


def test_what_is_not_to_be_had_is_asked_for_once(monkeypatch):
    """The device has room for less than was asked for: every size is tried once, the next calls begin
    with the one that was to be had, and the whole is asked for again after a while."""
    device = torch.device("cpu", 0)
    per_head = _tiles(1000, 1000, 1) * TILE
    asked, room = [], 3 * per_head + 8 * 4 * 1000

    def empty(size, **kw):
        asked.append(size)
        if size > room:
            raise torch.cuda.OutOfMemoryError("no")
        return size

    monkeypatch.setattr(ops.torch, "empty", empty)
    monkeypatch.setattr(ops, "_score_gradient_limits", {})
    monkeypatch.setattr(ops, "SCORE_GRADIENT_RETRY", 3)
    get = lambda **kw: ops._backward_scratch(1, 8, 1000, 1000, True, device, ops._score_gradient_limit(0), **kw)[1] // per_head
    assert get() == 2 and [a // per_head for a in asked] == [8, 4, 2]
    asked.clear()
    assert [get() for _ in range(3)] == [2, 2, 2] and [a // per_head for a in asked] == [2, 2, 2]
    asked.clear()
    assert get(refused=True) == 2 and [a // per_head for a in asked] == [4, 2]     # (the native entry asked for all)
    room = 0
    with pytest.raises(torch.cuda.OutOfMemoryError):       # not even delta
        get()
    assert ops._score_gradient_limit(1) == ops.SCORE_GRADIENT_BYTES                # another device


def _full_device():
    cuda = torch.device("cuda", 0)
    g = torch.Generator(device=cuda).manual_seed(2)
    q, k, v, dy = (torch.randn(1, 32, 2048, 128, generator=g, device=cuda).bfloat16() for _ in range(4))
    out, lse = ops.fused_attention(q, k, v, 0.1, causal=True, return_lse=True)
    want = ops.fused_attention_backward(q, k, v, out, lse, dy, 0.1, causal=True)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    whole = rt.load().ixb_fa_bwd_scratch_bytes(1, 32, 2048, 2048, 1, 1 << 40)
    total = torch.cuda.get_device_properties(0).total_memory
    # room for the three gradients and two thirds of dS
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + 3 * q.numel() * 2 + whole * 2 // 3 + (8 << 20)) / total)
    for calls in (1, 2):
        got = ops.fused_attention_backward(q, k, v, out, lse, dy, 0.1, causal=True)
        refusals = torch.cuda.memory_stats()["num_ooms"]
        assert refusals == 1, refusals
        assert all(torch.equal(a, e) for a, e in zip(got, want))
        del got
    assert ops._score_gradient_limits[0][0] == whole // 2


@pytest.mark.gpu
def test_backward_on_a_full_device(cuda):
    """The allocator may not grow by what dS takes, and refuses it once: the same gradients, in launches of
    fewer heads.  (In a process of its own: what other tests have left in the cache could hold dS.)"""
    here = os.path.dirname(os.path.abspath(__file__))
    code = f"import sys; sys.path[:0] = [{os.path.dirname(here)!r}, {here!r}]; import test_attention_scratch as t; t._full_device()"
    child = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert child.returncode == 0, child.stderr[-2000:]


@pytest.mark.gpu
def test_scratch_is_not_filled_under_deterministic_algorithms(cuda):
    """Torch then fills what it allocates: the three gradients, which the call returns, and nothing else; the
    bits are the same."""
    from torch.profiler import ProfilerActivity, profile

    g = torch.Generator(device=cuda).manual_seed(4)
    q, k, v, dy = (torch.randn(1, 4, 512, 128, generator=g, device=cuda).bfloat16() for _ in range(4))
    out, lse = ops.fused_attention(q, k, v, 0.1, causal=True, return_lse=True)
    want = ops.fused_attention_backward(q, k, v, out, lse, dy, 0.1, causal=True)
    was = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(True)
    try:
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            got = ops.fused_attention_backward(q, k, v, out, lse, dy, 0.1, causal=True)
            torch.cuda.synchronize()
    finally:
        torch.use_deterministic_algorithms(was)
    kernels = {e.key: e.count for e in p.key_averages() if e.device_time_total > 0}
    assert sum(n for name, n in kernels.items() if "fa_bwd" in name) == 3
    assert sum(n for name, n in kernels.items() if "fa_bwd" not in name) == 3, kernels
    assert all(torch.equal(a, e) for a, e in zip(got, want))
