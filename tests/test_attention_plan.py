"""How the attention forward goes about a call, which does not show in its results."""
import ctypes
import os
import subprocess
import sys

import pytest

from inductor_x_b200 import runtime as rt


def plan(b, h, sq, sk, causal=1):
    heads, blocks = ctypes.c_int32(-1), ctypes.c_int32(-1)
    assert rt.load().ixb_fa_fwd_plan(b, h, sq, sk, causal, ctypes.byref(heads), ctypes.byref(blocks)) == rt.IXB_OK
    return heads.value, blocks.value


def heads_together(*sizes, **mask):
    return plan(*sizes, **mask)[0]


@pytest.mark.parametrize("sq", [257, 300, 384])
def test_three_query_tiles_go_in_groups_of_eight_where_their_blocks_are_alike(sq):
    assert heads_together(4, 32, sq, sq) == heads_together(2, 4, sq, sq) == 8
    for sk in (sq + 1, 385, 1000):      # a block of two tiles has more products than the one before it in the order
        assert heads_together(4, 32, sq, sk) == 128     # K and V of all heads stay in L2
    assert heads_together(4, 32, sq, 4000) == 19        # groups of 40 MB, equal ones
    assert heads_together(4, 32, sq, sq, causal=0) == 1


def test_other_numbers_of_tiles():
    assert heads_together(4, 32, 256, 256) == heads_together(4, 32, 385, 385) == 128
    assert heads_together(8, 32, 4096, 4096) == 20 and heads_together(2, 8, 20000, 20000) == 8
    assert rt.load().ixb_fa_fwd_plan(0, 1, 1, 1, 1, *[ctypes.byref(ctypes.c_int32())] * 2) == rt.IXB_ERR_ARG


# the environment's word is taken where a kernel exists for it: no cluster of three or sixteen
@pytest.mark.parametrize("value,blocks", [("0", 0), ("8", 8), ("3", None), ("16", None), ("-4", None)])
def test_forced_sizes(value, blocks):
    code = ("import ctypes, sys; lib = ctypes.CDLL(sys.argv[1]); n = ctypes.c_int32()\n"
            "for h in (1, 16, 40, 112):\n"
            "    assert lib.ixb_fa_fwd_plan(1, h, 1, 2879, 0, ctypes.byref(n), ctypes.byref(n)) == 0; print(n.value)")

    def chosen(**env):
        return subprocess.run([sys.executable, "-c", code, rt.LIB_PATH], env=dict(os.environ, **env), capture_output=True,
                              text=True, check=True).stdout.split()

    assert chosen(IXB_FA_SPLIT=value) == (chosen() if blocks is None else [str(blocks)] * 4)


@pytest.mark.gpu
def test_heads_whose_blocks_all_run_at_once(cuda):
    assert heads_together(1, 32, 1024, 4096) == heads_together(4, 8, 1000, 3000) == 8
    assert heads_together(1, 32, 2048, 2048) == 32


@pytest.mark.gpu
def test_clusters_of_every_size_are_taken(cuda):
    blocks = {(h, sq, sk): plan(1, h, sq, sk)[1] for h in (1, 16, 40, 112, 320) for sq, sk in ((1, 2879), (3, 300), (300, 700))}
    assert blocks[1, 1, 2879] == 8 and blocks[16, 1, 2879] == 4 and blocks[40, 1, 2879] == 2 and blocks[112, 1, 2879] == 1
    assert blocks[1, 300, 700] == 4 and blocks[16, 300, 700] == 2 and blocks[40, 300, 700] == 1 and blocks[320, 300, 700] == 0


@pytest.mark.gpu
def test_the_first_call_of_a_process_may_be_captured(cuda):
    """What the choice asks of the device it may ask while a stream is being captured."""
    code = ("import torch; from inductor_x_b200 import ops\n"
            "q, k, v = (torch.randn(1, 4, s, 128, device='cuda', dtype=torch.bfloat16) for s in (3, 900, 900))\n"
            "torch.cuda.synchronize(); g = torch.cuda.CUDAGraph()\n"
            "with torch.cuda.graph(g): out = ops.fused_attention(q, k, v, 0.1, causal=False)\n"
            "g.replay(); assert torch.equal(out, ops.fused_attention(q, k, v, 0.1, causal=False)); print('captured')")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert out.stdout.split()[-1:] == ["captured"], out.stderr[-2000:]
