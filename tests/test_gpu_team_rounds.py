"""Team form with the rounds of its groups in straight-line code: team sizes
that give full, partial and single rounds, and groups left as loops."""

import numpy as np
import pytest

import hyk
from hyk import var
from hyk import workloads as W

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "oss": lambda n: (W.oss_sys(), W.oss_ics(n, seed=21)[0], None, 700.0),
    "kepler_var": lambda n: (var.var_ode_sys(W.kepler_sys(), var.var_args.vars, order=1), W.kepler_ics(n, seed=22), None,
                             0.4),
    "cr3bp": lambda n: (W.cr3bp_sys(),) + W.cr3bp_ics(n, seed=23) + (2.0,),
}


@pytest.mark.parametrize("team", [2, 4, 8, 16, 32])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_team_sizes_bitwise(oracle, name, team):
    n = 21
    sys_, st, pars, tf = SYSTEMS[name](n)
    ta = hyk.taylor_adaptive_batch(sys_, st, pars=pars, tol=1e-15, team_size=team)
    ta.propagate_until(tf)
    full, osys = st, sys_
    if name == "kepler_var":
        full, osys = np.concatenate([st, sys_.initial_variational_state(n)]), sys_.sys
    o = oracle.Oracle(osys, full, pars=pars, order=ta.order, mode=1)
    r = o.propagate_until(tf)
    assert np.array_equal(np.asarray(ta.state), o.state)
    assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy(), r["n_steps"].astype(np.int64))
