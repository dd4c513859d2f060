"""The event root finder against a plain restatement of its method (every
Bernstein coefficient of every interval, bisection from the interval's ends):
the same roots, bit for bit, for random polynomials, roots at and next to
dyadic numbers, double and clustered roots, wanted directions and ranges."""

import ctypes

import numpy as np
import pytest

_libm = ctypes.CDLL("libm.so.6")
_libm.fma.argtypes, _libm.fma.restype = [ctypes.c_double] * 3, ctypes.c_double
fma = _libm.fma


def _q(a, s):
    r = a[-1]
    for c in a[-2::-1]:
        r = fma(r, s, c)
    return r


def _find(g, h, s_lo, s_hi, direction, first_only):
    p = len(g) - 1
    a, hp = [], 1.0
    for x in g:
        a.append(x * hp)
        hp *= h
    bt = [[0.0] * (p + 1) for _ in range(p + 1)]
    for k in range(p + 1):
        for i in range(k + 1):
            r = 1.0
            for j in range(i):
                r = r * ((k - j) / (p - j))
            bt[k][i] = r
    hs = (h > 0) - (h < 0)
    out, d, i, scale = [], 0, 0, 1.0
    while True:
        lo, hi = i * scale, (i + 1) * scale
        if lo >= s_hi:
            break
        if hi > s_lo:
            c = list(a)
            for k in range(p):
                for j in range(p - 1, k - 1, -1):
                    c[j] = fma(c[j + 1], lo, c[j])
            wk = 1.0
            for k in range(p + 1):
                c[k] *= wk
                wk *= scale
            v, last = 0, 0
            for k in range(p + 1):
                acc = c[0] * bt[k][0]
                for j in range(1, k + 1):
                    acc = fma(bt[k][j], c[j], acc)
                sg = (acc > 0) - (acc < 0)
                if sg:
                    v += last != 0 and sg != last
                    last = sg
            if v >= 2 and d < 40:
                d, i, scale = d + 1, 2 * i, scale * 0.5
                continue
            if v >= 1:
                left, right, root = lo, hi, -1.0
                fl, fr = _q(a, left), _q(a, right)
                if fr == 0:
                    root = right
                elif fl != 0 and (fl < 0) != (fr < 0):
                    while True:
                        m = left + 0.5 * (right - left)
                        if not left < m < right:
                            break
                        fm = _q(a, m)
                        if fm == 0:
                            left = right = m
                            break
                        if (fm < 0) == (fl < 0):
                            left, fl = m, fm
                        else:
                            right = m
                    root = left + 0.5 * (right - left)
                if s_lo < root <= s_hi:
                    dq = p * a[p]
                    for n in range(p - 1, 0, -1):
                        dq = fma(dq, root, n * a[n])
                    sg = ((dq > 0) - (dq < 0)) * hs
                    if direction in (0, sg):
                        out.append((root, sg))
                        if first_only:
                            return out
        while d > 0 and i & 1:
            i, d, scale = i >> 1, d - 1, scale * 2
        if d == 0:
            break
        i += 1
    return out


def _poly(rng, kind, p):
    if kind == "decaying":
        return rng.normal(size=p + 1) * 0.6 ** np.arange(p + 1)
    roots = {"roots": rng.uniform(-0.5, 1.5, 4), "dyadic": rng.integers(1, 64, 3) / 64.0,
             "double": np.repeat(rng.uniform(0.1, 0.9, 2), 2), "cluster": rng.uniform(0.2, 0.8) + rng.uniform(0, 1e-6, 3),
             "near zero": rng.uniform(0.0, 1e-9, 1), "away": rng.uniform(-2.0, -0.01, 4)}[kind]
    c = np.polynomial.polynomial.polyfromroots(roots) * rng.normal()
    tail = np.zeros(p + 1)
    tail[: len(c)] = c
    return tail


@pytest.mark.parametrize("kind", ["decaying", "roots", "dyadic", "double", "cluster", "near zero", "away"])
def test_roots_equal_plain_bisection(oracle, kind):
    rng = np.random.default_rng(len(kind))
    found = 0
    for k in range(60):
        p = int(rng.integers(5, 25))
        g = _poly(rng, kind, p)
        h = float(rng.choice([1.0, -1.0, 0.37, -2.5]))
        g = g / h ** np.arange(p + 1)
        lo = float(rng.choice([0.0, 0.0, 0.25]))
        hi = float(rng.choice([1.0, 1.0, 0.7]))
        direction, first = int(rng.integers(-1, 2)), bool(rng.integers(0, 2))
        s, sg, _ = oracle.ev_find(g, h, lo, hi, direction, first)
        want = _find([float(x) for x in g], h, lo, hi, direction, first)
        assert [float(x) for x in s] == [w[0] for w in want] and [int(x) for x in sg] == [w[1] for w in want]
        found += len(want)
    assert found > 0 or kind == "away"

