"""Powers of polynomials in time, whose higher orders are zero: the recurrence
forms its products plainly (the integer products are for normal numbers only and
would be formed in vain at every order), with the oracle's bits."""

import ctypes

import numpy as np
import pytest

import hyk
from hyk import _lib
from hyk import workloads as W
from hyk.decompose import taylor_decompose


def _systems():
    x, y, z = hyk.make_vars("x", "y", "z")
    t, p = hyk.time, hyk.par[0]
    return {  # whether a power keeps its integer products (lane form, teams)
        "time": ([(x, (1.0 + t) ** -1.5 * x), (y, -y)], False, False),
        "square": ([(x, (2.0 + (1.0 + t) * (0.5 - t)) ** 2.5 * 0.01 - x), (y, hyk.square(1.0 + t) ** -1.5 * y)], False, False),
        "drift": ([(x, y**-1.5), (y, z), (z, 0.0 * z + p)], False, False),  # (z: linear in time only as far as is seen)
        "moving": ([(x, y**-1.5 - x), (y, p)], False, False),
        "mixed": ([(x, (1.0 + t) ** -1.5 + (1.0 + x * x) ** -1.5), (y, (1.0 + y * y) ** -1.5)], True, None),
        "states": ([(x, (1.0 + y * x) ** -1.5), (y, -x)], True, True),
        "kepler": (W.kepler_sys(), True, True),
    }


@pytest.mark.parametrize("team", [0, 2])
@pytest.mark.parametrize("name", [k for k in _systems() if k != "drift"])
def test_which_powers_use_integer_products(libhyk, name, team):
    sys_, lane, teams = _systems()[name]
    want = teams if team else lane
    d, keep = taylor_decompose(sys_).as_c()
    cfg = _lib.hyk_config_t(0, 0, 0, team)
    buf = ctypes.create_string_buffer(1 << 24)
    assert libhyk.hyk_codegen_check(ctypes.byref(d), 12, ctypes.byref(cfg), 2, buf, len(buf), None, None) == 0
    src = buf.value.decode()
    if want is not None:
        assert (" = HYK_MULK(" in src or "HYK_FMA(HYK_MULK(" in src) == want
    if name == "mixed" and not team:  # one of the two in x, and the one in y
        assert src.count("unsigned bad") == 2 * 10


@pytest.mark.gpu
@pytest.mark.parametrize("team", [1, 2, 8])
@pytest.mark.parametrize("name", list(_systems()))
def test_bitwise(oracle, name, team):
    sys_ = _systems()[name][0]
    n = 65
    st = np.random.default_rng(8).uniform(0.6, 1.4, (len(sys_), n))
    pars = np.random.default_rng(9).uniform(0.1, 0.3, (1, n)) if name in ("drift", "moving") else None
    ta = hyk.taylor_adaptive_batch(sys_, st, pars=pars, tol=1e-12, team_size=team)
    ta.propagate_until(0.4)
    o = oracle.Oracle(sys_, st, pars=pars, order=ta.order, mode=1)
    o.propagate_until(0.4)
    assert np.array_equal(np.asarray(ta.state), o.state)


@pytest.mark.gpu
def test_small_batch_of_powers_of_time_stays_in_the_lane_form():
    x, y = hyk.make_vars("x", "y")
    sys_ = [(x, (1.0 + hyk.time) ** -1.5 * y), (y, -x * (2.0 + hyk.time) ** -0.5)]
    ta = hyk.taylor_adaptive_batch(sys_, np.ones((2, 1000)))
    assert ta.module_info["team_size"] == 1
