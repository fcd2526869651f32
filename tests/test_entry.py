"""The module that calls the kernels' entry points: every argument arrives as it was given, and wrong ones are refused."""
import ctypes

import pytest
import torch

from esp_b200.csrc import ops
from esp_b200.csrc.build import load_entry, signature_letters
from esp_b200.errors import Backend


@pytest.fixture(scope="module")
def entry():
    m = load_entry(ops._SIGNATURES)
    m.set_careful_ptr(ops._careful_ptr)
    return m


@pytest.mark.parametrize("name", sorted(ops._SIGNATURES))
def test_every_entry_point_gets_its_arguments(entry, name):
    """A callback of the entry point's own C type stands in for it."""
    types = ops._SIGNATURES[name]
    given = []
    for i, t in enumerate(types):
        given.append({ctypes.c_void_p: (1 << 40) + i, ctypes.c_int: -1000 - i, ctypes.c_longlong: -(1 << 40) - i,
                      ctypes.c_ulonglong: (1 << 63) + i, ctypes.c_float: 0.25 + i}[t])
    got = []
    back = ctypes.CFUNCTYPE(ctypes.c_int, *types)(lambda *a: got.append(list(a)) or 7)
    f = entry.bind(ctypes.cast(back, ctypes.c_void_p).value, signature_letters(types))
    assert f(*given) == 7 and got == [given]


def test_conversions_and_refusals(entry):
    got = []
    back = ctypes.CFUNCTYPE(ctypes.c_int, *ops._SIGNATURES["esp_softcap"])(lambda *a: got.append(a) or -3)      # P q f P
    f = entry.bind(ctypes.cast(back, ctypes.c_void_p).value, "PqfP")
    assert f(None, True, 3, 0) == -3 and got == [(None, 1, 3.0, None)]
    for wrong in ((1, 2), (1, 2, "x", 3), (1, 2.5, 1.0, 3), (torch.ones(1), 1, 1.0, 0)):
        with pytest.raises(TypeError):
            f(*wrong)
    with pytest.raises(ValueError):
        entry.bind(1, "fffffPPP")
    assert len(got) == 1


def test_addresses_are_given_for_what_is_in_order_only(entry):
    assert entry.ptr(None) is None and entry.ptr(None, torch.float32, "x") is None
    with pytest.raises(Backend, match="x must live on the GPU"):
        entry.ptr(torch.ones(3), torch.float32, "x")
    with pytest.raises(AttributeError):
        entry.ptr(3.5)


def test_without_the_module_the_kernels_are_called_through_ctypes(monkeypatch):
    """Where it cannot be compiled (no g++, no headers) the entry points are reached as they were before there was a module."""
    got = []
    types = ops._SIGNATURES["esp_softcap"]
    back = ctypes.CFUNCTYPE(ctypes.c_int, *types)(lambda *a: got.append(a) or -3)

    def fails(signatures):
        raise Backend("g++ was not found")

    class Library:
        esp_softcap = back

    monkeypatch.setattr(ops, "load_entry", fails)
    monkeypatch.setattr(ops, "load_library", lambda name: Library)
    monkeypatch.setattr(ops, "_bound", {})
    monkeypatch.setattr(ops, "_entry", None)
    monkeypatch.setattr(ops, "_ptr", ops._careful_ptr)
    with pytest.warns(RuntimeWarning, match="g\\+\\+ was not found"):
        f = ops._fn("core", "esp_softcap")
    assert f(None, 1, 3.0, 1 << 40) == -3 and got == [(None, 1, 3.0, 1 << 40)]
    assert ops._fn("core", "esp_softcap") is f and ops._ptr is ops._careful_ptr
    with pytest.raises(Backend, match="no entry point"):
        ops._fn("core", "esp_depth_mix")


@pytest.mark.gpu
def test_addresses_of_tensors_on_the_device(entry):
    t = torch.ones(4, 6, device="cuda:0")
    assert entry.ptr(t) == entry.ptr(t, torch.float32) == entry.ptr(t[1:], ops.FLOATS, "x") - 24 == t.data_ptr()
    with pytest.raises(Backend, match="x must be contiguous"):
        entry.ptr(t.t(), torch.float32, "x")
    with pytest.raises(Backend, match="x has dtype"):
        entry.ptr(t, torch.bfloat16, "x")
    with pytest.raises(Backend, match="tensor has dtype"):
        entry.ptr(t.int(), ops.FLOATS)
