"""The entry points with arguments converted in C++ (dromos_b200._calls) answer as the ctypes functions behind them: the same
results, the same refusals of arguments. Calls of no rows, and sizes, need no GPU."""

import ctypes
import os
import sysconfig

import pytest
import torch

from dromos_b200 import abi, build, host

if abi._calls is None and not os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")):
    pytest.skip("no Python headers: the module cannot be built here", allow_module_level=True)


def test_the_module_is_there():
    assert abi._calls is not None, "not built (python -m dromos_b200.build)"


@pytest.fixture()
def lib():
    return abi.Library(abi.default_library_path())


def outcome(f, args):
    try:
        return f(*args)
    except Exception as e:  # noqa: BLE001 - which exception is what is compared
        return type(e), str(e)


WEIGHT = abi.make_weight(abi.W_BF16, torch.zeros(64, dtype=torch.uint8))
ADDRESSES = [None, 0, 64, 2**63 + 8, -8, ctypes.c_void_p(64), ctypes.c_void_p(None), b"bytes", "text", 1.5, object()]
WEIGHTS = [None, abi.WeightRef(WEIGHT), ctypes.byref(WEIGHT), ctypes.pointer(WEIGHT), WEIGHT, 64, ctypes.c_void_p(64)]
NUMBERS = [0, 7, -1, True, 2**31 + 5, 2**63, 2**70, 1.0, None, "1", ctypes.c_int(3)]
FLOATS = [0.5, 1, None, "1", ctypes.c_float(2.0), float("nan"), 1e300]


def gemv_args(**kw):  # M = 0: answers before anything is read
    a = dict(x=64, x_dtype=1, ld_x=64, w=abi.WeightRef(WEIGHT), bias=None, bias_dtype=1, y=64, y_dtype=0, ld_y=64, M=0, N=64, K=64, alpha=1.0, beta=0.0, stream=None)
    assert set(kw) <= set(a)
    a.update(kw)
    return tuple(a.values())


@pytest.mark.parametrize("name,values", [("x", ADDRESSES), ("w", WEIGHTS), ("ld_x", NUMBERS), ("N", NUMBERS), ("alpha", FLOATS), ("stream", ADDRESSES)])
def test_every_kind_of_argument(lib, name, values):
    fast, slow = lib.lx_gemv_w, lib.fn("lx_gemv_w")
    assert type(fast) is not type(slow)
    for v in values:
        args = gemv_args(**{name: v})
        assert outcome(fast, args) == outcome(slow, args), (name, v)


def test_counts_of_arguments_and_names(lib):
    fast, slow = lib.lx_gemm_workspace_bytes, lib.fn("lx_gemm_workspace_bytes")
    for args in ((), (1,), (9, 4096), (9, 4096, 0), (70, 512, 2), (9, 4096, 0, 5)):
        assert outcome(fast, args) == outcome(slow, args), args
    with pytest.raises(TypeError):
        fast(9, 4096, maths=0)
    assert fast.restype is slow.restype and fast.argtypes == slow.argtypes
    assert lib.lx_bf16x_row_bytes(4096) == 6192 and lib.lx_bf16x_row_bytes(0) == -1  # a 64-bit result with its sign


def test_the_callables_pass_for_ctypes_functions(lib):
    fast, slow = lib.lx_gemm_workspace_bytes, lib.fn("lx_gemm_workspace_bytes")
    assert ctypes.cast(fast, ctypes.c_void_p).value == ctypes.cast(slow, ctypes.c_void_p).value
    assert ctypes.CFUNCTYPE(ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.c_int)(ctypes.cast(fast, ctypes.c_void_p).value)(9, 4096, 0) == slow(9, 4096, 0)
    with pytest.raises(AttributeError):
        fast.no_such_attribute


def test_attributes_that_are_set_count(lib):
    seen = []
    want = lib.lx_gemm_workspace_bytes(9, 4096, 0)
    lib.lx_gemm_workspace_bytes.errcheck = lambda result, f, args: seen.append((result, args)) or -result
    assert lib.lx_gemm_workspace_bytes(9, 4096, 0) == -want and seen == [(want, (9, 4096, 0))]
    lib.lx_bf16x_row_bytes.restype = ctypes.c_int8
    assert lib.lx_bf16x_row_bytes(4096) == ctypes.c_int8(6192).value
    lib.lx_gemv_w.argtypes = None
    assert lib.lx_gemv_w.argtypes is None
    with pytest.raises(TypeError):
        lib.lx_gemv_w.argtypes = 5


def test_a_weight_reference_is_as_byref_has_it():
    ref = host.StoredWeight(abi.W_BF16, torch.zeros(64, dtype=torch.uint8)).ref()
    assert ref._obj is ref.struct
    assert ctypes.cast(ref, ctypes.POINTER(abi.LxWeight)).contents.data == ref.struct.data
    assert ctypes.cast(ref, ctypes.c_void_p).value == ctypes.cast(ctypes.byref(ref.struct), ctypes.c_void_p).value == ref.address


def test_a_weight_follows_its_struct():
    a, b = torch.zeros(64, dtype=torch.uint8), torch.zeros(64, dtype=torch.uint8)
    w = host.StoredWeight(abi.W_BF16, a)
    first = w.ref()
    assert w.ref() is first and first.address == ctypes.addressof(w.struct)
    w.struct = abi.make_weight(abi.W_BF16, b)
    assert w.ref().address == ctypes.addressof(w.struct)


def test_without_the_module_ctypes_converts(monkeypatch):
    monkeypatch.setattr(abi, "_calls", None)
    lib = abi.Library(abi.default_library_path())
    assert lib.lx_gemv_w is lib.fn("lx_gemv_w") and lib.lx_gemv_w(*gemv_args()) == 0


@pytest.mark.parametrize("compiler", ["false", "/no/such/compiler"])
def test_a_build_without_the_module_is_no_error(monkeypatch, tmp_path, capsys, compiler):
    module = tmp_path / os.path.basename(build.CALLS)
    module.write_bytes(b"of other sources")
    monkeypatch.setattr(build, "CALLS", str(module))
    monkeypatch.setenv("CXX", compiler)
    build.build_calls(stale=True)
    assert not module.exists() and "not built" in capsys.readouterr().err
