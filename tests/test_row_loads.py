"""How rows that start off a 16-byte boundary are read.  Row kernels are launched as dependents of
the kernel before them, and generated ones write in place, so their rows must not be read through
the path for data that nobody writes while the kernel runs."""
import os
import re

import pytest

IXB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inductor_x_b200", "csrc", "ixb")


@pytest.mark.parametrize("header,function", [("gen.cuh", r"void fetch_row\(const U\* rowp, RawRowU<"),
                                             ("row.cuh", r"void fetch\(const T\* base, int i, uint4 \(&words\)\[2\]\)")])
def test_covering_words_are_ordinary_loads(header, function):
    with open(os.path.join(IXB, header)) as f:
        text = f.read()
    body = text[re.search(function, text).end():]
    body = body[:body.index("\n  }\n")]
    assert "ldg_shared_word(" in body and not re.search(r"ldg_keep|__ldg|\.nc", body)
    with open(os.path.join(IXB, "common.cuh")) as f:
        load = re.search(r"uint4 ldg_shared_word\(.*?\n}", f.read(), re.S).group(0)
    assert 'asm volatile("ld.global.v4.u32' in load
