"""The reverse sweep's order-0 reciprocals: every slot it reads one from was
written by the forward recurrences, in both arithmetics, and the gradient of a
step (state and parameters) equals that of central differences for operations
of variables, of the time and of constants."""

import ctypes
import re
import subprocess

import numpy as np
import pytest

import hyk
from hyk import _lib
from hyk import workloads as W
from hyk.decompose import taylor_decompose

ORDER = 8


def _systems():
    x, y = hyk.make_vars("x", "y")
    p, t = hyk.par, hyk.time
    return {
        "variables": [(x, hyk.log(x) / y + hyk.sqrt(y)), (y, x**-1.5 - y**0.3 / x)],
        "constants": [(x, x * (p[0] / p[1]) + hyk.sqrt(p[0]) * y), (y, hyk.log(p[1]) * x - p[0] ** 1.5 / y)],
        "numbers": [(x, 2.0 / y - x / 3.0), (y, x / p[0] + p[1] / x)],
        "time": [(x, x / (1.0 + t) - hyk.sqrt(2.0 + t)), (y, hyk.log(1.5 + t) * y + (1.0 + t) ** -1.5 * x)],
        "kepler": W.kepler_sys(),
    }


def _source(libhyk, sys_, flags, verbose):
    d, keep = taylor_decompose(sys_).as_c()
    cfg = _lib.hyk_config_t(0, 0, _lib.HYK_CFG_ADJOINT | flags, 0)
    buf = ctypes.create_string_buffer(1 << 24)
    rc = libhyk.hyk_codegen_check(ctypes.byref(d), ORDER, ctypes.byref(cfg), verbose, buf, len(buf), None, None)
    assert rc == 0, libhyk.hyk_last_error()
    return buf.value.decode()


@pytest.mark.parametrize("flags", [0, _lib.HYK_CFG_PIN_ARITH])
@pytest.mark.parametrize("name", list(_systems()))
def test_gradient_of_a_step(libhyk, tmp_path, name, flags):
    sys_ = _systems()[name]
    src = _source(libhyk, sys_, flags, 3)
    for i, s in re.findall(r"const double (i\d+) = (S\[\d+ \* HYK_STRIDE\]);", src):
        assert "{} = {};".format(s, i) in src, (i, s)
    f, so = str(tmp_path / "h.cpp"), str(tmp_path / "h.so")
    with open(f, "w") as fh:
        fh.write(src)
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", f, "-o", so], check=True)
    H = ctypes.CDLL(so)
    n, npar = len(sys_), taylor_decompose(sys_).n_pars
    x0, pars = np.array([1.1, 0.8, 0.3, 0.1, 0.7, 0.2][:n]), np.array([0.7, 1.3])
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    t0, h = ctypes.c_double(0.4), ctypes.c_double(0.05)
    S = np.full(H.hyk_host_nslot(), 7.5)  # (nothing may depend on what the slots held)

    def step(x, p):
        x, p, x1 = np.ascontiguousarray(x), np.ascontiguousarray(p), np.zeros(n)
        H.hyk_host_step(ptr(S), ptr(x), ptr(p), t0, h, ptr(x1))
        return x1

    l0 = np.random.default_rng(0).normal(size=n)
    lam, pb = l0.copy(), np.zeros(2)
    H.hyk_host_adjoint(ptr(S), ptr(x0), ptr(pars), t0, h, ptr(lam), ptr(pb))
    e = 1e-6
    fd = np.array([l0 @ (step(x0 + e * v, pars) - step(x0 - e * v, pars)) for v in np.eye(n)]) / (2 * e)
    assert np.max(np.abs(lam - fd)) < 1e-8 * np.max(np.abs(fd))
    fp = np.array([l0 @ (step(x0, pars + e * v) - step(x0, pars - e * v)) for v in np.eye(2)[:npar]]) / (2 * e)
    assert np.all(np.abs(pb[:npar] - fp) < 1e-8 * max(1.0, np.max(np.abs(fp), initial=0.0)))
