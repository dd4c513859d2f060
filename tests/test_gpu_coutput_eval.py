"""Continuous output evaluated in one launch: rows inside, between, at and
outside the lanes' steps, forward and backward, both precisions, equal to the
stored coefficients evaluated on the host."""

import numpy as np
import pytest

import hyk
from hyk import workloads as W

pytestmark = pytest.mark.gpu


def _host(co, t):
    """Horner with fused multiply-adds in the precision of the output, the step
    chosen per lane by its start times."""
    import ctypes

    tcs, times = np.asarray(co.tcs), np.asarray(co.times)
    lo = co._tlo.cpu().numpy()
    f32 = tcs.dtype == np.float32
    libm = ctypes.CDLL("libm.so.6")
    fma = libm.fmaf if f32 else libm.fma
    ty = ctypes.c_float if f32 else ctypes.c_double
    fma.argtypes, fma.restype = [ty] * 3, ty
    k, dim, p1, B = tcs.shape
    R = tcs.dtype.type
    out = np.empty((t.shape[0], dim, B), tcs.dtype)
    for r in range(t.shape[0]):
        for b in range(B):
            sgn = R(-1) if times[-1, b] < times[0, b] else R(1)
            keys = times[:k, b] * sgn
            i = min(max(int(np.searchsorted(keys, t[r, b] * sgn, side="right")) - 1, 0), k - 1)
            ah, bh, bl = t[r, b], times[i, b], lo[i, b]
            s = ah - bh
            bb = s - ah
            e = (ah - (s - bb)) + ((-bh) - bb)
            dt = R(s + R(e + (R(0) - bl)))
            for j in range(dim):
                acc = tcs[i, j, -1, b]
                for n in range(p1 - 2, -1, -1):
                    acc = R(fma(float(acc), float(dt), float(tcs[i, j, n, b])))
                out[r, j, b] = acc
    return out


@pytest.mark.parametrize("back", [False, True])
@pytest.mark.parametrize("n", [1, 3, 129])
@pytest.mark.parametrize("fp", [np.float64, np.float32])
def test_rows_bitwise(fp, n, back):
    st = W.kepler_ics(n, seed=17).astype(fp)
    ta = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-9 if fp == np.float64 else 1e-6,
                                   fp_type=float if fp == np.float64 else np.float32)
    tf = np.linspace(1.0, 2.5, n).astype(fp) * fp(-1.0 if back else 1.0)
    co, _ = ta.propagate_until(tf, c_output=True)
    times = np.asarray(co.times)
    rows = [tf * fp(u) for u in (-0.1, 0.0, 0.3, 0.9999, 1.0, 1.2)] + [times[0], times[1], times[-1]]
    t = np.ascontiguousarray(np.stack(rows).astype(fp))
    want = _host(co, t)
    got = co(t)
    assert got.shape == want.shape and np.array_equal(got, want)
    assert np.array_equal(co.output, want[-1])
    assert np.array_equal(co(t[2]), want[2]) and np.array_equal(co.output, want[2])
    assert co(t[:0]).shape == (0, 6, n)


def test_tape_and_records_that_outgrow_their_store(oracle):
    """More steps than the first store holds: resumed with the same results."""
    n = 5000  # 5000 lanes: 111 records of the Kepler coefficients in 512 MiB
    st = W.kepler_ics(n, seed=18)
    ta = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15)
    co, _ = ta.propagate_until(8.0, c_output=True)
    tb = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15)
    tb.propagate_until(8.0)
    assert np.array_equal(np.asarray(ta.state), np.asarray(tb.state))
    assert co.n_steps == int(tb.propagate_res_tensors["n_steps"].max()) and co.n_steps > 111
