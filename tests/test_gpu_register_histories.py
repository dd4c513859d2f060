"""Lane form with the histories in registers: orders on both sides of the most
values it holds, every operation kind, both precisions, events included."""

import numpy as np
import pytest

import hyk
from hyk import workloads as W

pytestmark = pytest.mark.gpu


def ops():
    x, y = hyk.make_vars("x", "y")
    return [(x, hyk.exp(-y) - hyk.par[0] * x), (y, hyk.sqrt(x) * hyk.cos(hyk.time) / (1.0 + y))]


def powers():
    x, y = hyk.make_vars("x", "y")
    return [(x, hyk.log(y) * x**-1.5), (y, -x * (x * x + y * y) ** 0.3)]


@pytest.mark.parametrize("tol", [1e-3, 1e-9, 1e-16, 1e-17, 1e-18, 1e-19])
@pytest.mark.parametrize("name", ["pendulum", "kepler", "ops", "powers"])
def test_orders_bitwise(oracle, name, tol):
    n, rng, pars = 75, np.random.default_rng(5), None
    if name == "pendulum":
        sys_, st = W.pendulum_sys(), W.pendulum_ics(n, seed=1)
    elif name == "kepler":
        sys_, st = W.kepler_sys(), W.kepler_ics(n, seed=2)
    else:
        sys_, st = (ops() if name == "ops" else powers()), rng.uniform(1.0, 1.5, (2, n))
        pars = rng.uniform(0.1, 0.3, (1, n)) if name == "ops" else None
    for mode in ("persistent", "plain"):
        ta = hyk.taylor_adaptive_batch(sys_, st, pars=pars, tol=tol, prop_mode=mode, team_size=1)
        tf = np.linspace(0.3, 0.8, n)
        ta.propagate_until(tf)
        o = oracle.Oracle(sys_, st, pars=pars, order=ta.order, mode=1)
        r = o.propagate_until(tf)
        # (log(y) x^-1.5 leaves the reals on one of the lanes: not-a-number on both sides)
        assert np.array_equal(np.asarray(ta.state), o.state, equal_nan=True)
        assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy(), r["n_steps"].astype(np.int64))
    ta.step(write_tc=True)
    o.step()
    assert np.array_equal(np.asarray(ta.state), o.state, equal_nan=True)


@pytest.mark.parametrize("tol", [1e-4, 1e-7, 1e-10])
@pytest.mark.parametrize("name", ["pendulum", "kepler"])
def test_float_orders_bitwise(oracle, name, tol):
    n = 777
    sys_, st = ((W.pendulum_sys(), W.pendulum_ics(n, seed=3)) if name == "pendulum" else
                (W.kepler_sys(), W.kepler_ics(n, seed=4)))
    st = st.astype(np.float32)
    ta = hyk.taylor_adaptive_batch(sys_, st, tol=tol, fp_type=np.float32)
    ta.propagate_until(2.0)
    o = oracle.Oracle(sys_, st.astype(np.float64), order=ta.order, mode=1, prec=2)
    r = o.propagate_until(2.0)
    assert np.array_equal(np.asarray(ta.state).astype(np.float64), o.state)
    assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy(), r["n_steps"].astype(np.int64))
