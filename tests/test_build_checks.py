"""Checks that the build makes on what the compiler reports."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inductor_x_b200", "csrc")


@pytest.mark.skipif(shutil.which("make") is None, reason="make not available")
@pytest.mark.parametrize("regs,ok", [((168, 168), True), ((168, 160), False), ((166, 168), False), ((168,), False), ((), False)])
def test_attention_forward_with_another_register_count_does_not_build(tmp_path, regs, ok):
    """The register split between its warpgroups adds up to the count at launch."""
    log = tmp_path / "ptxas.log"
    other = "ptxas info    : Compiling entry function '_Z5otherv' for 'sm_100a'\nptxas info    : Used 32 registers\n"
    log.write_text(other + "".join(f"ptxas info    : Compiling entry function '_Z13fa_fwd_kernelILb{i}EEv' for 'sm_100a'\n"
                                   f"ptxas info    : Used {r} registers, used 1 barriers\n" for i, r in enumerate(regs)) + other)
    out = subprocess.run(["make", "-s", "-C", CSRC, "check_regs", f"LOG={log}"], capture_output=True, text=True)
    assert (out.returncode == 0) is ok, out.stdout + out.stderr
    assert ok or "the register split needs 168" in out.stdout
