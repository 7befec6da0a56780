"""Calls into C entry points without ctypes, against ctypes itself (no GPU needed)."""
import ctypes

import pytest
import torch

from from_scratch_inference_engine_b200.csrc import build

I, LL, F, P = ctypes.c_int, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p


def module():
    compiled = build.host_call()
    if compiled is build._PlainCalls:
        pytest.skip("no headers of this Python")
    return compiled


# integers in registers and on the stack, floats before, between and behind them, as many as there may be
@pytest.mark.parametrize("kinds", [[I], [P, I, LL, F], [F] * 8, [P] * 7 + [F] + [I] * 5 + [LL, F, P], [LL] * 48,
                                   [P, F] * 8 + [I] * 40])
def test_arguments_arrive(kinds):
    got = []
    callback = ctypes.CFUNCTYPE(I, *kinds)(lambda *args: (got.append(args), -7)[1])
    tensor = torch.zeros(3)
    values, want = [], []
    for n, kind in enumerate(kinds):
        if kind is F:
            values.append(0.37 * n - 1)
            want.append(ctypes.c_float(0.37 * n - 1).value)
        elif kind is P and n % 3 == 1:
            values.append(None)
            want.append(None)
        elif kind is P and n % 3 == 2:
            values.append(tensor)
            want.append(tensor.data_ptr())
        else:
            value = {I: -n - 1, LL: -(1 << 40) - n, P: (1 << 47) + n}[kind]
            values.append(value)
            want.append(value)
    signature = "".join("f" if kind is F else "i" for kind in kinds)
    address = ctypes.cast(callback, P).value
    call = module().Function(address, signature, "entry")
    assert call(*values) == -7 and got.pop() == tuple(want)
    with pytest.raises(TypeError):
        call(*values[:-1])
    with pytest.raises(TypeError):
        call(*values, 1)
    with pytest.raises((TypeError, AttributeError)):
        call(*values[:-1], "text")
    assert not got


def test_what_is_refused():
    for signature in ("p", "i" * 49, "f" * 9):
        with pytest.raises(ValueError):
            module().Function(1, signature, "entry")
    assert module().fits(torch.zeros(2), None, False) is False                 # not on the GPU


@pytest.mark.parametrize("plain", [False, True])
def test_a_library_of_calls(plain, monkeypatch):
    """The C library's own functions: those with declared arguments of the known types, through the module and without it."""
    if plain:
        monkeypatch.setattr(build, "_host_call", build._PlainCalls)
    lib = ctypes.CDLL(None)
    lib.abs.argtypes, lib.abs.restype = [I], I
    lib.memcmp.argtypes, lib.memcmp.restype = [P, P, LL], I
    lib.atof.argtypes, lib.atof.restype = [P], ctypes.c_double
    calls = build.fast_calls(lib)
    assert calls.abs(-5) == 5
    a, b = torch.arange(4), torch.tensor([0, 1, 2, 9])
    assert calls.memcmp(a, b, 24) == 0 and calls.memcmp(a, b, 32) != 0
    assert calls.atof is lib.atof                                              # its result is no int
