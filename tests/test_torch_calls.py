"""The native form of the device calls (csrc/torch_calls.cpp) without a GPU: whatever torch refuses comes back as a Python
exception, whatever the library declines as W8A8Error, and what is not a torch tensor goes through ctypes."""
import numpy as np
import pytest
import torch

from volvoxai_b200 import w8a8

calls = pytest.importorskip("volvoxai_b200._torch_calls")


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
