"""How the blocks of the attention kernels end.  A wait that gives up must not let a block go while
copies into its shared memory or products on it are under way.  The wait cannot be made to run out
without a kernel built for it, so this reads the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inductor_x_b200", "csrc")


@pytest.mark.parametrize("source,kernel", [("fa_fwd.cu", "fa_fwd_kernel"), ("fa_bwd.cu", "fa_bwd_dkv_kernel"),
                                           ("fa_bwd.cu", "fa_bwd_dq_kernel")])
def test_roles_wait_for_what_they_started(source, kernel):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    body = text[re.search(rf"\b{kernel}\(const __grid_constant__", text).end():]
    body = body[:body.index("\n}\n")]
    # every barrier that a copy completes on is waited for at the end of the role that started it
    loaded = set(re.findall(r"mbar_arrive_expect_tx\(&(\w+)", body))
    awaited = set(re.findall(r"await_copies<\w+>\(&?(\w+), ", body))
    assert loaded and loaded <= awaited
    assert body.count("await_products(&drained)") == 1 and "mbar_init(&drained, 1)" in body
    if "request_next_block(" in body:
        assert "await_copies<2>(next_full, asked)" in body


@pytest.mark.parametrize("source,kernel", [("fa_split.cu", "fa_split_kernel"), ("fa_bwd.cu", "fa_bwd_dq_ds_kernel")])
def test_roles_with_a_barrier_for_each_slot_do_too(source, kernel):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    body = text[re.search(rf"\b{kernel}\(const __grid_constant__", text).end():]
    body = body[:body.index("\n}\n")]
    loaded = set(re.findall(r"mbar_arrive_expect_tx\(&(\w+)", body))
    awaited = set(re.findall(r"await_copies<\w+>\(&?(\w+)(?:\[\w+\])?, ", body))
    assert loaded and loaded <= awaited
    assert body.count("await_products(&drained)") == 1 and "mbar_init(&drained, 1)" in body
    if "request_next_block(" in body:
        assert "await_copies<2>(next_full, asked)" in body


def test_these_waits_are_bounded_and_ignore_the_abort_flag():
    with open(os.path.join(CSRC, "ixb", "tcgen05.cuh")) as f:
        text = f.read()
    for name, wait in (("await_copies", "mbar_wait(&full[last % STAGES], (last / STAGES) & 1);"),
                       ("await_products", "mbar_wait(bar, 0)")):
        body = text[re.search(rf"void {name}\(", text).end():]
        assert wait in body[:body.index("\n}\n")]
