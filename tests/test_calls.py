"""The module of frequent entry points against the ctypes signatures: same functions, same status codes, the argument forms that the
mirror passes.  No device: a NULL context answers NotInitialized after its arguments have been taken."""
import ctypes as C

import pytest

NOT_INITIALIZED = 8


@pytest.fixture(scope="module")
def calls():
    from ferrograd_b200 import _lib, build
    build.build()
    return _lib.calls()


def entries(calls):
    return [n for n in dir(calls) if n.startswith("fg_")]


def test_every_function_takes_what_the_library_takes(calls):
    from ferrograd_b200 import _lib
    assert len(entries(calls)) >= 20
    for name in entries(calls):
        args = _lib.SIGNATURES[name][1]
        zero = [0.0 if a is C.c_float else 0 if a in (C.c_uint32, C.c_uint64, C.c_int32) else None for a in args]
        assert getattr(calls, name)(*zero) == getattr(_lib.load(), name)(*zero) == NOT_INITIALIZED, name
        for wrong in (zero[:-1], zero + [0]):
            with pytest.raises(TypeError):
                getattr(calls, name)(*wrong)


def test_argument_forms(calls):
    class Thing:
        ptr = 4096

    class Bad:
        ptr = "x"

    for p in (None, 0, 4096, Thing(), C.c_void_p(4096), C.c_void_p(None)):
        assert calls.fg_softmax_fwd(0, 1, 1, p, p) == NOT_INITIALIZED
    assert calls.fg_sgd_step(C.c_void_p(None), None, None, 3, 1, 1.0, True) == NOT_INITIALIZED
    for bad in (Bad(), "x", object()):
        with pytest.raises((TypeError, ValueError)):
            calls.fg_softmax_fwd(0, 1, 1, bad, None)
    with pytest.raises(TypeError):
        calls.fg_softmax_fwd(0, 1.5, 1, None, None)
    with pytest.raises(TypeError):
        calls.fg_sgd_step(None, None, None, 3, "x", 1.0, True)


def test_programs(calls):
    from ferrograd_b200.backend import EW
    assert calls.OPS == EW
    prog = [("input", 0, 0, 0.0), (EW["input"], 1, 0, 0), ["add", 0, 1, 0.0]]
    assert calls.chain_fwd(None, 0, 4, prog, [1, None], 2, None) == NOT_INITIALIZED
    assert calls.chain_fwd(None, 0, 4, tuple(prog), (1, 2), 2, [None, 3, None]) == NOT_INITIALIZED
    assert calls.chain_bwd(None, 0, 4, prog, [1, 2], 3, [None], False) == NOT_INITIALIZED
    assert calls.chain_fwd(None, 0, 4, [], [], None, None) == NOT_INITIALIZED
    for bad, error in (([("sqrt", 0, 0, 0.0)], KeyError), ([("add", 0, 0)], ValueError), ([3], TypeError), (3, TypeError), ([("add", "x", 0, 0.0)], TypeError)):
        with pytest.raises(error):
            calls.chain_fwd(None, 0, 4, bad, [1], 2, None)
    with pytest.raises(ValueError):
        calls.chain_fwd(None, 0, 4, prog, [1, 2], 2, [None])
    with pytest.raises(IndexError):
        calls.chain_bwd(None, 0, 4, prog, [1, 2], 3, [1, 2, 3], False)


@pytest.mark.parametrize("accumulate", [True, 1, 1.0, "1"])
@pytest.mark.parametrize("numpy_type", [None, "bool_", "int64", "float32"])
def test_the_mirror_takes_what_int_takes(calls, accumulate, numpy_type):
    # flags go through int(), as they did with the foreign-function calls; no device: the answer to a NULL context
    import numpy as np

    from ferrograd_b200 import FgError, GpuContext, _lib
    ctx = GpuContext.__new__(GpuContext)
    ctx.lib, ctx.handle, ctx._c, ctx._h = _lib.load(), None, calls, 0
    flag = accumulate if numpy_type is None else getattr(np, numpy_type)(int(accumulate))
    prog = [("input", 0, 0, 0.0), ("neg", 0, 0, 0.0)]
    for call in (lambda: ctx.eltwise_chain_bwd(prog, [16], 16, [16], 4, accumulate=flag), lambda: ctx.softmax_bwd(16, 16, 16, 1, 1, accumulate=flag),
                 lambda: ctx.sgd_step(16, 16, 1, 0.1, zero_grad=flag), lambda: ctx.gemm(16, 16, 16, 1, 1, 1, transA=flag, transB=flag)):
        with pytest.raises(FgError) as e:
            call()
        assert e.value.code == NOT_INITIALIZED
