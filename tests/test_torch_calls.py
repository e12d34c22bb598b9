"""The native form of the device calls (csrc/torch_calls.cpp) without a GPU: whatever torch refuses comes back as a Python
exception, whatever the library declines as W8A8Error, and what is not a torch tensor goes through ctypes."""
import os
import subprocess

import numpy as np
import pytest
import torch

from volvoxai_b200 import build, w8a8

if not build.torch_calls_built():
    pytest.skip("_torch_calls.so is not built for this Python and torch", allow_module_level=True)
from volvoxai_b200 import _torch_calls as calls  # noqa: E402  (a module that does not load fails here)


class Closed:
    """A context whose handle has been given back."""
    _h = 0


@pytest.mark.parametrize("x,error", [(torch.tensor(1.0), IndexError), (torch.zeros(2, 8).to_sparse(), RuntimeError),
                                     (np.zeros((2, 8), np.float32), TypeError), (None, TypeError)])
def test_inputs_that_torch_refuses_raise(x, error):
    with pytest.raises(error):
        calls.linear_f32(0, 0, x, 8, None, 0)


def test_arguments_that_do_not_fit_raise():
    x = torch.zeros(2, 8)
    with pytest.raises(TypeError):
        calls.linear_f32(0, 0, x)
    with pytest.raises(TypeError):
        calls.linear_f32("ctx", 0, x, 8, None, 0)
    with pytest.raises(RuntimeError):
        calls.linear_f32(0, 0, x, -5, None, 0)
    with pytest.raises(TypeError):
        calls.quantize_linear(0, x, "scale", 0, 0)
    with pytest.raises(RuntimeError):
        torch.vmap(lambda v: calls.linear_f32(0, 0, v, 8, None, 0))(torch.zeros(3, 2, 8))


def test_a_declined_call_raises_the_library_error():
    """Null handles are declined by every entry before anything is touched."""
    x = torch.zeros(2, 8)
    weight = Closed()
    weight.d_out = 8
    for call in (lambda: w8a8.Context.linear_f32(Closed, weight, x), lambda: w8a8.Context.linear_i8(Closed, weight, x, 0.1),
                 lambda: w8a8.Context.linear_f32_fused(Closed, weight, x, residual=x),
                 lambda: w8a8.Context.rmsnorm_linear_f32_fused(Closed, weight, x, x[0], 1e-6),
                 lambda: w8a8.Context.qlinear_device(Closed, weight, x.to(torch.int8), 0.1, 0, 0.1, 0),
                 lambda: w8a8.Context.quantize_linear(Closed, x, 0.1), lambda: w8a8.Context.dequantize_linear(Closed, x.to(torch.uint8), 0.1),
                 lambda: w8a8.Context.requantize_linear(Closed, x.to(torch.int8), 0.1, 0, 0.1, 0)):
        with pytest.raises(w8a8.W8A8Error) as e:
            call()
        assert e.value.code == 0 and "null argument" in str(e.value)


def test_only_torch_tensors_take_the_native_form():
    assert w8a8._calls(torch.zeros(1)) is calls
    assert w8a8._calls(torch.nn.Parameter(torch.zeros(1))) is calls
    assert w8a8._calls(np.zeros(1)) is None and w8a8._calls(None) is None


class Memory:
    """Not a torch tensor, but with a device pointer and a row pitch."""
    def __init__(self, at=0, pitch=8):
        self.at, self.pitch = at, pitch

    def data_ptr(self):
        return self.at

    def stride(self, dim):
        return self.pitch


def test_calls_with_other_memory_go_through_ctypes():
    """An output, residual, norm weight or norm output that is not torch's: declined by the library here (null handles),
    where the native form would refuse the argument."""
    x, other = torch.zeros(2, 8), Memory()
    context, weight = Closed(), Closed()
    weight.d_out, context._L, context.handle, weight.handle = 8, w8a8._lib.load(), None, None
    f = w8a8.Context
    for call in (lambda: f.linear_f32(context, weight, x, out=other), lambda: f.linear_i8(context, weight, x, 0.1, out=other),
                 lambda: f.linear_f32_fused(context, weight, x, residual=other), lambda: f.linear_f32_fused(context, weight, x, out=other),
                 lambda: f.rmsnorm_linear_f32_fused(context, weight, x, other, 1e-6),
                 lambda: f.rmsnorm_linear_f32_fused(context, weight, x, x[0], 1e-6, norm_out=other),
                 lambda: f.rmsnorm_linear_f32_fused(context, weight, x, None, 1e-6)):
        with pytest.raises(w8a8.W8A8Error):
            call()
    assert w8a8._calls(x, None, x) is calls and w8a8._calls(x, None, other) is None


@pytest.fixture
def scratch(tmp_path, monkeypatch):
    """build.py with the module elsewhere, and w8a8.py as before its first call."""
    monkeypatch.setattr(build, "TORCH_CALLS", str(tmp_path / "_torch_calls.so"))
    monkeypatch.setattr(w8a8, "_torch_calls", False)
    return tmp_path


def put(scratch, key):
    (scratch / "_torch_calls.so").write_bytes(b"...built for " + key.encode() + b"\0...")


def test_the_library_builds_where_the_module_cannot(scratch, monkeypatch, capsys):
    put(scratch, "another")
    monkeypatch.setattr(subprocess, "run", lambda *a, **k: subprocess.CompletedProcess(a, 1, "", "no Python.h"))
    assert build.build_torch_calls() is None and "no Python.h" in capsys.readouterr().err
    assert os.listdir(scratch) == []
    def missing(*a, **k):
        raise FileNotFoundError("g++")
    monkeypatch.setattr(subprocess, "run", missing)
    assert build.build_torch_calls(force=True) is None
    assert w8a8._calls(torch.zeros(1)) is None


@pytest.mark.parametrize("same", [True, False])
def test_a_module_for_another_torch_is_not_used(scratch, monkeypatch, same):
    put(scratch, build.torch_calls_key())
    if not same:
        monkeypatch.setattr(torch, "__version__", "0.1")
    assert build.torch_calls_built() == same
    assert (w8a8._calls(torch.zeros(1)) is calls) == same
    built = []
    os.utime(build.TORCH_CALLS)
    monkeypatch.setattr(subprocess, "run", lambda *a, **k: built.append(a) or subprocess.CompletedProcess(a, 0, "", ""))
    build.build_torch_calls()
    assert bool(built) != same and build.torch_calls_built() == same      # (the stand-in compiler leaves no module)
