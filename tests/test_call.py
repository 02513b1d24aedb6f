"""The extension module in front of ribn_gemv (csrc/call.c): what it hands over and what it refuses.  No GPU: the function it calls is a
Python callback, or ribn_gemv itself without a context."""
import ctypes
import types

import pytest
import torch

import engine_b200
from engine_b200 import _lib

ENTRY = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64,
                         ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64, ctypes.c_uint32)


@pytest.fixture
def entry():
    calls = []

    @ENTRY
    def function(*arguments):
        calls.append(arguments)
        return 5

    function.calls = calls
    function.address = ctypes.cast(function, ctypes.c_void_p).value
    return function


def test_arguments_arrive_as_ribn_gemv_takes_them(entry):
    gemv = _lib.load_call().gemv
    x, y = torch.zeros(3, 64, dtype=torch.bfloat16), torch.zeros(3, 7)
    assert gemv(entry.address, 4096, 12, 8192, x, y, 3) == 5
    assert entry.calls == [(4096, 12, 8192, x.data_ptr(), _lib.RIBN_BF16, 192, y.data_ptr(), _lib.RIBN_F32, 21, 3)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.float64, torch.int32])
@pytest.mark.parametrize("which", [0, 1])
def test_other_dtypes_are_refused_before_the_call(entry, dtype, which):
    tensors = [torch.zeros(64), torch.zeros(64)]
    tensors[which] = tensors[which].to(dtype)
    with pytest.raises(TypeError, match="float32 or bfloat16"):
        _lib.load_call().gemv(entry.address, 4096, 12, 8192, *tensors, 1)
    assert not entry.calls


def test_what_is_not_a_tensor_or_a_number_is_refused(entry):
    gemv = _lib.load_call().gemv
    x = torch.zeros(64)
    raising = types.SimpleNamespace(dtype=torch.float32, data_ptr=lambda: 1 / 0, numel=lambda: 64)
    odd = types.SimpleNamespace(dtype=torch.float32, data_ptr=lambda: "here", numel=lambda: 64)
    for arguments, error in (((4096, 12, 8192, None, x, 1), AttributeError), ((4096, 12, 8192, x, raising, 1), ZeroDivisionError),
                             ((4096, 12, 8192, odd, x, 1), TypeError), (("context", 12, 8192, x, x, 1), TypeError),
                             ((4096, -1, 8192, x, x, 1), OverflowError), ((4096, 12, 8192, x, x, "one"), TypeError), ((4096, 12, 8192, x, x), TypeError)):
        with pytest.raises(error):
            gemv(entry.address, *arguments)
    assert not entry.calls


def test_a_closed_context_is_an_error_not_a_crash():
    context = engine_b200.RibnContext.__new__(engine_b200.RibnContext)   # as close() leaves one
    context._lib = _lib.load()
    context.handle, context._address = None, 0
    context._gemv_address = ctypes.cast(context._lib.ribn_gemv, ctypes.c_void_p).value
    context._call_gemv = _lib.load_call().gemv
    weight = types.SimpleNamespace(_descriptor_address=ctypes.addressof(_lib.QWeight()))
    with pytest.raises(engine_b200.CudaQuantizedKernelError) as e:
        engine_b200.CudaQ4KGemv.from_context(context).execute(weight, torch.zeros(256), torch.zeros(1))
    assert e.value.kind == "InvalidArgument"
