"""The team form's common group of state updates (right-hand sides with and
without a history, state variables, folded negations) and its common group of
sines and cosines: the oracle's bits for every team size."""

import numpy as np
import pytest

import hyk
from hyk import cos, sin

pytestmark = pytest.mark.gpu


def _systems():
    x, y, z, w = hyk.make_vars("x", "y", "z", "w")
    return {
        # a state variable, its negation, a product, a negated product
        "signs": [(x, -y), (y, x), (z, x * w), (w, -(y * z))],
        # sines and cosines as leads and followers, negated, of two arguments
        "trig": [(x, sin(y) * cos(z)), (y, -cos(x)), (z, -w), (w, sin(x) + cos(y))],
        "pair": [(x, cos(y)), (y, -sin(y)), (z, -x), (w, 0.5 * sin(z))],
    }


@pytest.mark.parametrize("team", [2, 4, 32])
@pytest.mark.parametrize("fp", [np.float64, np.float32])
@pytest.mark.parametrize("name", ["signs", "trig", "pair"])
def test_update_and_trig_groups_bitwise(oracle, name, fp, team):
    sys_ = _systems()[name]
    n = 37
    st = np.random.default_rng(5).normal(0.0, 0.7, (4, n)).astype(fp)
    ta = hyk.taylor_adaptive_batch(sys_, st, tol=1e-6 if fp is np.float32 else 1e-15, team_size=team, fp_type=fp)
    ta.propagate_until(1.5)
    one = hyk.taylor_adaptive_batch(sys_, st, tol=1e-6 if fp is np.float32 else 1e-15, team_size=1, fp_type=fp)
    one.propagate_until(1.5)
    assert np.array_equal(np.asarray(ta.state), np.asarray(one.state))
    if fp is np.float64:
        o = oracle.Oracle(sys_, st, order=ta.order, mode=1)
        o.propagate_until(1.5)
        assert np.array_equal(np.asarray(ta.state), o.state)
