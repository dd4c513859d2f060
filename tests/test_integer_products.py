"""Products of a coefficient and a small half-integer in integer arithmetic
(the power recurrence's n alpha - j (alpha + 1)): the bits of the double
product wherever the operand is in range, flagged where it is not, and the
recurrences around them equal to the oracle where operands are zero, tiny or
huge."""

import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

import hyk
from hyk import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_product_bits(tmp_path):
    src = tmp_path / "m.cpp"
    src.write_text('#include "hyk_dmath.h"\n'
                   'extern "C" void mulk(const double *b, unsigned k, long n, double *out, unsigned *bad) {\n'
                   '    for (long i = 0; i < n; ++i) { bad[i] = 0; out[i] = hyk_dm_mulk(b[i], k, bad + i); }\n}\n')
    so = str(tmp_path / "m.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "heyoka.py_gb300", "csrc"), str(src), "-o", so],
                   check=True)
    L = ctypes.CDLL(so)
    rng = np.random.default_rng(11)
    n = 20000
    u = rng.integers(0, 1 << 63, n, dtype=np.uint64) | (rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63))
    # runs of equal low bits (ties), every exponent, the ends of the range
    low = rng.integers(0, 53, n).astype(np.uint64)
    u[::3] &= ~((np.uint64(1) << low[::3]) - np.uint64(1))
    u[1::3] |= (np.uint64(1) << low[1::3]) - np.uint64(1)
    edge = np.array([0, 1, 63, 64, 65, 1963, 1964, 2046, 2047], dtype=np.uint64) << np.uint64(52)
    u[: 9 * 100] = (u[: 9 * 100] & np.uint64((1 << 52) - 1)) | np.repeat(edge, 100)
    b = u.view(np.float64)
    e = (u >> np.uint64(52)) & np.uint64(0x7FF)
    inside = (e >= 64) & (e < 1964)
    for num in list(range(1, 130)) + [255, 256, 511, 1023, 2047]:
        for sgn in (1.0, -1.0):
            coef = sgn * num / 2.0
            m, ex = math.frexp(abs(coef))
            kp = int(m * 2048)  # 1024 <= kp < 2048, |coef| = kp 2^(ex - 11)
            k = (((ex - 1) << 20) + ((1 << 31) if sgn < 0 else 0) + kp) & 0xFFFFFFFF
            out, bad = np.empty(n), np.empty(n, dtype=np.uint32)
            L.mulk(b.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint(k), ctypes.c_long(n), out.ctypes.data_as(ctypes.c_void_p),
                   bad.ctypes.data_as(ctypes.c_void_p))
            assert np.array_equal(bad == 0, inside)
            with np.errstate(all="ignore"):
                want = b * coef
            assert np.array_equal(out[inside].view(np.uint64), want[inside].view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("team", [1, 4])
@pytest.mark.parametrize("scale", [1e-150, 1.0, 1e150])
@pytest.mark.parametrize("alpha", [-0.5, 1.5, 2.5])
def test_power_out_of_range_bitwise(oracle, alpha, scale, team):
    x, y, z, u, v, w = hyk.make_vars("x", "y", "z", "u", "v", "w")
    # the first powers of the time in x^2 + y^2 + z^2 vanish exactly on the circular lanes
    f = (x * x + y * y + z * z) ** alpha
    c = scale if alpha == -0.5 else 1.0
    sys_ = [(x, u), (y, v), (z, w), (u, -c * x * f), (v, -c * y * f), (w, -c * z * f)]
    n = 64
    st = np.zeros((6, n))
    ph = np.linspace(0.0, 3.0, n)
    ph[: n // 2] = 0.0
    st[0], st[1] = scale * np.cos(ph), scale * np.sin(ph)
    st[3], st[4] = -scale * np.sin(ph), scale * np.cos(ph) * np.where(np.arange(n) < n // 4, 1.0, 1.1)
    ta = hyk.taylor_adaptive_batch(sys_, st, tol=1e-15, team_size=team)
    ta.propagate_until(0.8)
    o = oracle.Oracle(sys_, st, order=ta.order, mode=1)
    r = o.propagate_until(0.8)
    assert np.array_equal(np.asarray(ta.state), o.state, equal_nan=True)
    assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy(), r["n_steps"].astype(np.int64))


@pytest.mark.gpu
def test_planar_circular_kepler_bitwise(oracle):
    st = np.zeros((6, 32))
    st[0], st[4] = 1.0, 1.0
    for team in (1, 8):
        ta = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15, team_size=team)
        ta.propagate_until(7.0)
        o = oracle.Oracle(W.kepler_sys(), st, order=ta.order, mode=1)
        o.propagate_until(7.0)
        assert np.array_equal(np.asarray(ta.state), o.state)
