"""The step-size rule with one logarithm on the host: the bits of the rule with
two, for norms over the whole range of normal numbers (their quotients may
underflow), zero, subnormal and not finite ones, and close to where the two
logarithms are equal."""

import ctypes
import subprocess

import numpy as np
import pytest

from cuda_host import INTRINSICS
from hyk import _lib
from hyk import workloads as W
from hyk.decompose import taylor_decompose

BUILTINS = r"""
static const struct { unsigned x; } threadIdx = {0}, blockIdx = {0};
template <class T> static inline T atomicMin(T *p, T) { return *p; }
"""

DRIVER = r"""
extern "C" void rho(long n, const hyk_real *p, const hyk_real *q, const hyk_real *num, hyk_real *one, hyk_real *two) {
    for (long i = 0; i < n; ++i) {
        one[i] = hyk_rho_one(p[i], q[i], num[i]);
        two[i] = HYK_DM_RHO(p[i], q[i], num[i], HYK_INV_P, HYK_INV_PM1);
    }
}
"""


def _lib_of(libhyk, order, f32, tmp):
    d, keep = taylor_decompose(W.pendulum_sys()).as_c()
    cfg = _lib.hyk_config_t(0, 0, _lib.HYK_CFG_FLOAT32 if f32 else 0, 0)
    buf = ctypes.create_string_buffer(1 << 24)
    assert libhyk.hyk_codegen_check(ctypes.byref(d), order, ctypes.byref(cfg), 2, buf, len(buf), None, None) == 0
    # the definitions up to the end of the step-size rule
    src = buf.value.decode()
    end = src.index("#endif", src.index("hyk_rho_one(hyk_real m_p"))
    src = src[:end] + "#endif\n"
    f, so = str(tmp / "r.cpp"), str(tmp / "r.so")
    with open(f, "w") as fh:
        fh.write(INTRINSICS + BUILTINS + src + DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-shared", "-fPIC", f, "-o", so], check=True)
    return ctypes.CDLL(so)


def _both(lib, ty, p, q, num):
    out = [np.empty(len(p), ty), np.empty(len(p), ty)]
    keep = [np.ascontiguousarray(v, ty) for v in (p, q, num)]
    a = [v.ctypes.data_as(ctypes.c_void_p) for v in keep]
    lib.rho(ctypes.c_long(len(p)), *a, *[o.ctypes.data_as(ctypes.c_void_p) for o in out])
    return out


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("order", [2, 3, 9, 19, 41])
def test_bits_of_the_two_logarithm_rule(libhyk, tmp_path, order, f32):
    lib = _lib_of(libhyk, order, f32, tmp_path)
    ty = np.float32 if f32 else np.float64
    emin, emax = (-126.0, 127.0) if f32 else (-1022.0, 1023.0)
    rng, n = np.random.default_rng(order), 40000
    with np.errstate(all="ignore"):
        # any normal norms, num >= 1
        lp, ln = rng.uniform(emin, emax, n), rng.uniform(0.0, emax, n)
        lq = rng.uniform(emin, emax, n)
        # a third of them where the logarithms are equal or nearly so
        k = n // 3
        lq[:k] = np.clip((lp - ln)[:k] * (order - 1) / order + ln[:k] + rng.choice([0.0, 1e-9, 1e-3, 0.1, 1.0], k)
                         * rng.normal(size=k), emin, emax)
        # and a third where quotients underflow, next to each other
        m = slice(k, 2 * k)
        ln[m] = rng.uniform(0.7 * emax, emax, k)
        lp[m] = np.clip(ln[m] + (emin - 25.0) * rng.uniform(0.9, 1.1, k), emin, emax)
        lq[m] = np.clip(ln[m] + (lp[m] - ln[m]) * rng.uniform(0.9, 1.05, k), emin, emax)
        p, q, num = (np.exp2(v).astype(ty) for v in (lp, lq, ln))
        special = np.array([0.0, 5e-324, 1e-310, 1e-40, np.inf, np.nan, 1.0], ty)
        p, q = np.concatenate([p, np.repeat(special, 49)]), np.concatenate([q, np.tile(np.repeat(special, 7), 7)])
        num = np.concatenate([num, np.tile(np.where(special >= 1.0, special, 1.0), 49)]).astype(ty)
    num = np.where(num < 1, ty(1), num)
    one, two = _both(lib, ty, p, q, num)
    same = (one == two) | (np.isnan(one) & np.isnan(two))
    assert same.all(), list(zip(p[~same], q[~same], num[~same], one[~same], two[~same]))[:5]
