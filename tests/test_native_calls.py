"""Library entry points called from native code (csrc/host_launch.cpp): the same results and errors as the
Python functions they stand in for, which take every call that is out of the ordinary."""
import types

import pytest
import torch

from inductor_x_b200 import _ixb_host, ops
from inductor_x_b200 import runtime as rt

NAMES = ("rms_norm", "fused_attention", "fused_attention_backward")


class Tagged(torch.Tensor):
    pass


def test_what_is_out_of_the_ordinary_is_left_to_python():
    rt.load()
    x, w = torch.ones(4, 8), torch.ones(8)
    assert _ixb_host.rms_norm(x, w, 1e-6, None, False) is None                    # host memory
    assert _ixb_host.rms_norm(x.as_subclass(Tagged), w, 1e-6, None, False) is None
    assert _ixb_host.rms_norm(x, w, 1, None, False) is None and _ixb_host.rms_norm(x, w) is None
    assert _ixb_host.rms_norm(None, w, 1e-6, None, False) is None
    m = torch.empty(2, 2, 4, 128, device="meta", dtype=torch.float16)
    assert _ixb_host.fused_attention(m, m, m, 1.0, False, True) is None            # no memory
    assert _ixb_host.fused_attention_backward(m, m, m, m, m, m, 1.0, False, 1 << 30) is None
    with pytest.raises(ValueError):
        ops.rmsnorm(x, w)
    with pytest.raises(TypeError):
        _ixb_host.bind_library(1)


def _both(monkeypatch, call):
    """Results of the native route (which is checked to be the one taken) and of the Python route."""
    counts = rt.native_calls
    with monkeypatch.context() as m:
        m.setattr(rt, "check", lambda *a: pytest.fail("the Python route was taken"))
        native = call()
    assert rt.native_calls == counts + 1
    with monkeypatch.context() as m:
        m.setattr(ops, "_ixb_host", types.SimpleNamespace(**{n: lambda *a: None for n in NAMES}))
        python = call()
    assert rt.native_calls == counts + 2
    native, python = (r if isinstance(r, tuple) else (r,) for r in (native, python))
    assert len(native) == len(python)
    for a, b in zip(native, python):
        assert a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype and torch.equal(a, b)
        assert not a.requires_grad


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(16, 4096), (3, 161), (2, 3, 64), (7,), (0, 8)])
def test_rms_norm(cuda, monkeypatch, dtype, shape):
    rt.load()
    x, r = (torch.randn(*shape, device=cuda).to(dtype) for _ in range(2))
    w = torch.nn.Parameter(torch.randn(shape[-1], device=cuda).to(dtype))
    _both(monkeypatch, lambda: ops.rmsnorm(x, w, 1e-5))
    _both(monkeypatch, lambda: ops.rmsnorm(x, w, 1e-5, residual=r))
    _both(monkeypatch, lambda: ops.rmsnorm(x, w, 1e-5, residual=r, return_residual=True))
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
        _both(monkeypatch, lambda: ops.rmsnorm(x, w, 1e-5, residual=r))
        torch.cuda.current_stream().synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("bsnd", [False, True])
def test_attention(cuda, monkeypatch, causal, bsnd):
    rt.load()
    make = lambda s: (torch.randn(2, s, 3, 128, device=cuda).half().transpose(1, 2) if bsnd
                      else torch.randn(2, 3, s, 128, device=cuda).half())
    q, k, v, dy = make(70), make(200), make(200), make(70)
    _both(monkeypatch, lambda: ops.fused_attention(q, k, v, 0.1, causal=causal))
    _both(monkeypatch, lambda: ops.fused_attention(q, k, v, 0.1, causal=causal, return_lse=True))
    out, lse = ops.fused_attention(q, k, v, 0.1, causal=causal, return_lse=True)
    _both(monkeypatch, lambda: ops.fused_attention_backward(q, k, v, out, lse, dy, 0.1, causal=causal))
    monkeypatch.setattr(ops, "SCORE_GRADIENT_BYTES", 0)
    _both(monkeypatch, lambda: ops.fused_attention_backward(q, k, v, out, lse, dy, 0.1, causal=causal))


@pytest.mark.gpu
def test_errors_are_what_they_were(cuda):
    rt.load()
    x, w = torch.ones(4, 8, device=cuda), torch.ones(8, device=cuda)
    for bad in (lambda: ops.rmsnorm(x.t(), w), lambda: ops.rmsnorm(x, w[:4]), lambda: ops.rmsnorm(x, w.half()),
                lambda: ops.rmsnorm(x, w, residual=x.half()), lambda: ops.rmsnorm(x, w.cpu())):
        with pytest.raises(ValueError):
            bad()
    with pytest.raises(rt.IxbError) as e:
        ops.rmsnorm(torch.ones(4, 0, device=cuda), torch.ones(0, device=cuda))
    assert e.value.status == rt.IXB_ERR_ARG
    q = torch.zeros(1, 1, 8, 128, dtype=torch.bfloat16, device=cuda)
    with pytest.raises(rt.IxbError):
        ops.fused_attention(q, q, q, -1.0)
    with pytest.raises(ValueError):
        ops.fused_attention(q, q[..., :64], q, 1.0)
    with pytest.raises(RuntimeError):      # a batched tensor has no memory of its own
        torch.vmap(lambda t: ops.rmsnorm(t, w))(x.unsqueeze(0).repeat(2, 1, 1))


@pytest.mark.gpu
def test_dispatch_modes_see_what_python_would_show_them(cuda, monkeypatch):
    """A mode that raises, one that counts the operations, a fake-tensor mode with real operands: the same
    error or the same operations with and without the native entries."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        def __init__(self, raises=False):
            super().__init__()
            self.ops, self.raises = [], raises

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.ops.append(str(func))
            if self.raises:
                raise KeyError("not here")
            return func(*args, **(kwargs or {}))

    rt.load()
    x, w = torch.ones(4, 8, device=cuda), torch.ones(8, device=cuda)
    q = torch.ones(1, 1, 8, 128, dtype=torch.bfloat16, device=cuda)
    lse = torch.ones(1, 1, 8, device=cuda)
    calls = (lambda: ops.rmsnorm(x, w, residual=x, return_residual=True), lambda: ops.fused_attention(q, q, q, 1.0, return_lse=True),
             lambda: ops.fused_attention_backward(q, q, q, q, lse, q, 1.0))

    def outcome(make, call):
        mode = make()
        with mode:
            try:
                call()
                out = None
            except Exception as e:
                out = type(e)
        return out, getattr(mode, "ops", None)

    for call in calls:
        for make in (Seen, lambda: Seen(True), lambda: FakeTensorMode(allow_non_fake_inputs=True)):
            with_native = outcome(make, call)
            with monkeypatch.context() as m:
                m.setattr(ops, "_ixb_host", types.SimpleNamespace(**{n: lambda *a: None for n in NAMES}))
                assert outcome(make, call) == with_native
        assert outcome(lambda: Seen(True), call)[0] is KeyError and outcome(Seen, call)[1]
    torch.cuda.synchronize()
