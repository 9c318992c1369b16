"""The native launch path of generated kernels: which calls go straight to the module's entry, and
that everything else reaches the general route with its arguments unchanged.  A module that only
records what it is given stands in for a kernel, so no GPU is needed."""
import ctypes
import subprocess
import threading

import pytest
import torch

from inductor_x_b200 import config
from inductor_x_b200.codegen import jit

RECORDER = r"""
static long long seen[8]; static int n, status;
int ixb_gen_launch(void** ptrs, const long long* ints, void* stream) {
  __sync_fetch_and_add(&n, 1); seen[0] = ints[0]; seen[1] = ints[1]; seen[2] = (long long)stream; return status; }
long long get(int i) { return i < 0 ? n : seen[i]; }
void set_status(int s) { status = s; }
"""


@pytest.fixture()
def kernel(tmp_path):
    src, so = tmp_path / "r.c", tmp_path / "r.so"
    src.write_text(RECORDER)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(so), str(src)], check=True)
    k = jit.GeneratedKernel("recorder", str(so), {"name": "recorder"})
    k.lib.get.restype = ctypes.c_longlong
    return k


def test_plain_calls_are_launched_natively(kernel):
    kernel.run(5, 1 << 40, stream=77)
    assert [kernel.lib.get(i) for i in (-1, 0, 1, 2)] == [1, 5, 1 << 40, 77]
    assert kernel.launches == kernel.run.launches == 1


def test_everything_else_takes_the_general_route(kernel, monkeypatch):
    calls = []
    k = jit._native_launcher()(lambda *a, **kw: calls.append((a, kw)) or "general", vars(config))
    t = torch.zeros(3)
    assert k(1, 2, stream=0) == "general"                # not bound to a module
    k.bind(ctypes.cast(kernel.fn, ctypes.c_void_p).value)
    assert k(1, t, stream=0) == "general"                # a host tensor
    assert k(1, True, stream=0) == "general"             # not exactly an int
    assert k(1, 1 << 70, stream=0) == "general"          # beyond 64 bits
    assert k(1, 2, stream=None) == "general" and k(1, 2) == "general"
    monkeypatch.setattr(config, "profile_bandwidth", True)
    assert k(1, 2, stream=0) == "general"
    monkeypatch.setattr(config, "profile_bandwidth", False)
    monkeypatch.setattr(config, "dry_run", True)
    assert k(1, 2, stream=0) == "general"
    monkeypatch.setattr(config, "dry_run", False)
    assert calls[1] == ((1, t), {"stream": 0}) and len(calls) == 8
    assert k(1, 2, stream=0) is None and kernel.lib.get(-1) == 1
    kernel.lib.set_status(1)                             # a launch that fails is worded by the general route
    assert k(1, 2, stream=0) == "general" and k.launches == 1


def test_failure_is_raised(kernel):
    kernel.lib.set_status(700)
    with pytest.raises(RuntimeError, match="cudaError 700"):
        kernel.run(1, 2, stream=0)


def test_failed_launch_is_not_tried_again(kernel):
    """Its status may be an earlier call's and the kernel may have run: an update in place would be
    applied twice."""
    kernel.lib.set_status(1)
    with pytest.raises(RuntimeError, match="cudaError 1"):
        kernel.run(1, 2, stream=0)
    assert kernel.lib.get(-1) == 1 and kernel.launches == 0
    seen = []
    k = jit._native_launcher()(lambda *a, **kw: seen.append((a, kw)), vars(config))
    k.bind(ctypes.cast(kernel.fn, ctypes.c_void_p).value)
    k(1, 2, stream=0)
    assert kernel.lib.get(-1) == 2 and seen == [((), {"status": 1})]


def test_pending_measurement_and_bounds_reports_are_not_passed_by(kernel):
    tuned = jit.GeneratedKernel("t", kernel.path, {"tune": dict(candidates=[(1,) * 6], idempotent=True, default=[1] * 6,
                                                                rows=1 << 20, row_bytes=1 << 10)})
    checked = jit.GeneratedKernel("b", kernel.path, {"bounds": True})
    for k in (tuned, checked):
        seen = []
        k.run = jit._native_launcher()(lambda *a, **kw: seen.append(a), vars(config))
        k._arm()
        k.run(1, 2, stream=0)
        assert seen == [(1, 2)]


def test_threads(kernel):
    def work():
        for _ in range(2000):
            kernel.run(1, 2, stream=3)

    ts = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert kernel.lib.get(-1) == 8000 and kernel.launches == 8000
