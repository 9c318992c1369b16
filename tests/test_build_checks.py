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


@pytest.mark.skipif(shutil.which("make") is None, reason="make not available")
def test_launch_extension_is_built_for_the_interpreter_and_the_torch_in_use():
    """Another torch release makes it out of date, and another interpreter looks for another file."""
    import sysconfig

    from inductor_x_b200 import _ixb_host

    tag = sysconfig.get_config_var("EXT_SUFFIX")
    assert _ixb_host.__file__.endswith(tag)

    def is_linked(tag, *given):
        out = subprocess.run(["make", "-n", "-C", CSRC, f"../_ixb_host{tag}", *given], capture_output=True, text=True, check=True)
        return "host_launch.cpp" in out.stdout

    assert is_linked(tag, "TORCH=9.9.9")
    assert is_linked(".cpython-399-x86_64-linux-gnu.so", "PYTAG=.cpython-399-x86_64-linux-gnu.so")
    if os.path.isdir(os.path.join(CSRC, "build")):  # (not kept everywhere that the built files are)
        assert not is_linked(tag)
