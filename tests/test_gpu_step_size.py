"""The step-size rule with one logarithm: the oracle's bits over many states,
at scales far from one, and where a norm is zero, subnormal or not finite."""

import numpy as np
import pytest

import hyk
from hyk import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("team", [1, 8])
def test_many_states_bitwise(oracle, team):
    st = W.kepler_ics(60000, seed=8)
    ta = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15, team_size=team)
    o = oracle.Oracle(W.kepler_sys(), st, order=ta.order, mode=1)
    for _ in range(3):
        ta.step()
        oc, h = o.step()
        assert np.array_equal(ta.last_h, h) and np.array_equal(np.asarray(ta.state), o.state)


@pytest.mark.parametrize("tol", [1e-3, 1e-9, 1e-16])
@pytest.mark.parametrize("scale", [0.0, 1e-320, 1e-305, 1e-160, 1e-30, 1.0, 1e30, 1e160, 1e300, np.inf])
def test_scales_bitwise(oracle, scale, tol):
    x, y, v, w = hyk.make_vars("x", "y", "v", "w")
    # the coefficients of (x, v) and (y, w) fall off at different rates
    sys_ = [(x, v), (v, -hyk.par[0] * x), (y, w), (w, hyk.par[1] * y)]
    rng = np.random.default_rng(3)
    n = 300
    st = scale * rng.uniform(-1.0, 1.0, (4, n)) if np.isfinite(scale) else np.full((4, n), np.inf)
    pars = np.exp(rng.uniform(-12.0, 12.0, (2, n)))
    for team in (1, 2):
        ta = hyk.taylor_adaptive_batch(sys_, st, pars=pars, tol=tol, team_size=team)
        ta.step()
        o = oracle.Oracle(sys_, st, pars=pars, order=ta.order, mode=1)
        oc, h = o.step()
        assert np.array_equal(ta.last_h, h, equal_nan=True)
        assert np.array_equal(np.asarray(ta.state), o.state, equal_nan=True)
