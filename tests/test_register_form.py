"""The lane form with the histories in registers: where it is taken, seen in
the source that hyk_codegen_check generates for the GPU, which compiles."""

import ctypes

import pytest

import hyk
from hyk import _lib
from hyk import workloads as W
from hyk.decompose import taylor_decompose


def _source(libhyk, sys_, order, flags=0, blk=0, compile_it=False):
    d, keep = taylor_decompose(sys_).as_c()
    cfg, ns = _lib.hyk_config_t(blk, 0, flags, 1), ctypes.c_uint32()
    buf = ctypes.create_string_buffer(1 << 24)
    rc = libhyk.hyk_codegen_check(ctypes.byref(d), order, ctypes.byref(cfg), 0 if compile_it else 2, buf, len(buf),
                                  ctypes.byref(ns), None)
    assert rc == 0, libhyk.hyk_last_error().decode() + buf.value.decode()
    return buf.value.decode(), ns.value


@pytest.mark.parametrize("flags,inreg", [(0, 1), (_lib.HYK_CFG_PIN_ARITH, 0), (_lib.HYK_CFG_ADJOINT, 0),
                                         (_lib.HYK_CFG_GLOBAL_JETS, 0), (_lib.HYK_CFG_NO_COLD_ROWS, 1),
                                         (_lib.HYK_CFG_FLOAT32, 1)])
def test_the_check_follows_the_module(libhyk, flags, inreg):
    src, ns = _source(libhyk, W.pendulum_sys(), 20, flags)
    assert "#define HYK_INREG {}\n".format(inreg) in src
    if inreg:
        assert ns == 2 * 21  # the rows only
    if flags & _lib.HYK_CFG_FLOAT32:
        assert "#define HYK_TPB 64\n" in src and "__launch_bounds__(HYK_TPB, " in src
    _source(libhyk, W.pendulum_sys(), 20, flags, compile_it=True)
