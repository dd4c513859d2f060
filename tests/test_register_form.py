"""The lane form with the histories in registers: where it is taken, seen in
the source that hyk_codegen_check generates for the GPU, which compiles."""

import ctypes

import numpy as np
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


def linear(n):
    x = hyk.make_vars(*["x{}".format(i) for i in range(n)])
    return [(x[i], -x[(i + 1) % n]) for i in range(n)]


@pytest.mark.parametrize("n,flags,inreg", [
    (2, 0, 1), (8, 0, 1),  # five warps' rows in the shared memory of an SM
    (9, 0, 0), (10, 0, 0), (9, _lib.HYK_CFG_NO_COLD_ROWS, 1),
    (24, _lib.HYK_CFG_FLOAT32, 1)])
def test_rows_that_leave_too_few_warps(libhyk, n, flags, inreg):
    src, ns = _source(libhyk, linear(n), 9 if flags & _lib.HYK_CFG_FLOAT32 else 20, flags)
    assert "#define HYK_INREG {}\n".format(inreg) in src
    assert ns == (n * (10 if flags & _lib.HYK_CFG_FLOAT32 else 21) if inreg else n)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["persistent", "plain"])
@pytest.mark.parametrize("n", [1, 8, 9, 10])
def test_linear_systems_bitwise(oracle, n, mode):
    sys_ = linear(n) if n > 1 else [(hyk.make_vars("x"), hyk.par[0] * hyk.make_vars("x"))]
    st = np.random.default_rng(n).uniform(0.5, 1.0, (n, 333))
    pars = np.random.default_rng(7).uniform(-1.0, -0.5, (1, 333)) if n == 1 else None
    ta = hyk.taylor_adaptive_batch(sys_, st, pars=pars, team_size=1, prop_mode=mode)
    tf = np.linspace(0.5, 9.0, 333)
    ta.propagate_until(tf)
    o = oracle.Oracle(sys_, st, pars=pars, order=ta.order, mode=1)
    o.propagate_until(tf)
    assert np.array_equal(np.asarray(ta.state), o.state)


@pytest.mark.gpu
def test_block_size_of_a_float_system_in_global_memory(oracle):
    """Short histories, but rows that leave room for fewer than four warps."""
    sys_ = linear(60)
    st = np.random.default_rng(4).uniform(0.5, 1.0, (60, 200)).astype(np.float32)
    ta = hyk.taylor_adaptive_batch(sys_, st, team_size=1, fp_type=np.float32)
    assert ta.module_info["smem_per_lane"] == 0 and ta.module_info["block_lanes"] == 128
    ta.propagate_until(3.0)
    o = oracle.Oracle(sys_, st.astype(np.float64), order=ta.order, mode=1, prec=2)
    o.propagate_until(3.0)
    assert np.array_equal(np.asarray(ta.state).astype(np.float64), o.state)


@pytest.mark.gpu
@pytest.mark.parametrize("fp", [np.float64, np.float32])
@pytest.mark.parametrize("name", ["pendulum", "linear"])
def test_coefficients_copied_from_registers(oracle, name, fp):
    """A step's coefficients, which outputs read from the shared memory."""
    sys_ = W.pendulum_sys() if name == "pendulum" else linear(4)
    st = np.random.default_rng(6).uniform(0.1, 1.0, (len(sys_), 99)).astype(fp)
    f32 = fp == np.float32
    ta = hyk.taylor_adaptive_batch(sys_, st, team_size=1, fp_type=np.float32 if f32 else float)
    ta.propagate_until(0.7)
    ta.step(write_tc=True)
    o = oracle.Oracle(sys_, st.astype(np.float64), order=ta.order, mode=1, prec=2 if f32 else 0)
    o.propagate_until(0.7)
    o.step()
    assert np.array_equal(np.asarray(ta.state).astype(np.float64), o.state)
    assert np.array_equal(np.asarray(ta.tc).astype(np.float64), o.tc)
