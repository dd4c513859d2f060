"""The kernel form chosen for a batch size: whatever it is, the oracle's bits."""

import numpy as np
import pytest

import hyk
from hyk import var
from hyk import workloads as W

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "kepler": lambda n: (W.kepler_sys(), W.kepler_ics(n, seed=61), None, 0.6),
    "cr3bp": lambda n: (W.cr3bp_sys(),) + W.cr3bp_ics(n, seed=62) + (1.5,),
    "oss": lambda n: (W.oss_sys(), W.oss_ics(n, seed=63)[0], None, 900.0),
    "kepler_var": lambda n: (var.var_ode_sys(W.kepler_sys(), var.var_args.vars, order=1), W.kepler_ics(n, seed=64), None,
                             0.4),
}


@pytest.mark.parametrize("n", [1, 37, 1216, 2500])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_form_of_batch_size_bitwise(oracle, name, n):
    sys_, st, pars, tf = SYSTEMS[name](n)
    ta = hyk.taylor_adaptive_batch(sys_, st, pars=pars, tol=1e-15)
    ta.propagate_until(tf)
    full, osys = st, sys_
    if name == "kepler_var":
        full, osys = np.concatenate([st, sys_.initial_variational_state(n)]), sys_.sys
    pick = np.unique(np.linspace(0, n - 1, 24).astype(np.int64))
    o = oracle.Oracle(osys, np.ascontiguousarray(full[:, pick]),
                      pars=None if pars is None else np.ascontiguousarray(pars[:, pick]), order=ta.order, mode=1)
    r = o.propagate_until(tf)
    assert np.array_equal(np.asarray(ta.state)[:, pick], o.state)
    assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy()[pick], r["n_steps"].astype(np.int64))


def test_form_named_by_the_caller_is_kept():
    st = W.kepler_ics(5, seed=65)
    lane = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15, team_size=1)
    team = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15, team_size=2)
    dbg = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15, debug=True)
    assert [t.module_info["team_size"] for t in (lane, team, dbg)] == [1, 2, 1]
