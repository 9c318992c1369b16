"""How the attention forward goes about a call, which does not show in its results."""
import ctypes

import pytest

from inductor_x_b200 import runtime as rt


def heads_together(b, h, sq, sk, causal=1):
    heads = ctypes.c_int32(-1)
    assert rt.load().ixb_fa_fwd_plan(b, h, sq, sk, causal, ctypes.byref(heads)) == rt.IXB_OK
    return heads.value


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
    assert rt.load().ixb_fa_fwd_plan(0, 1, 1, 1, 1, ctypes.byref(ctypes.c_int32())) == rt.IXB_ERR_ARG
