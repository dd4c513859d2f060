"""The host copies that an ensemble's generator gets: each its own integrator,
pickled with its own data only."""

import pickle

import numpy as np
import pytest

import hyk
from hyk import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_iter", [2, 300])
def test_pickled_copies(n_iter):
    ta = hyk.taylor_adaptive_batch(W.pendulum_sys(), np.full((2, 4), 0.1))
    sizes, back = [], []

    def gen(tac, i):
        tac.state[:] = 0.1 + 0.001 * i
        s = pickle.dumps(tac)
        sizes.append(len(s))
        if i == n_iter - 1:
            back.append(pickle.loads(s))
        return tac

    ret = hyk.ensemble_propagate_until_batch(ta, 1.0, n_iter, gen)
    assert max(sizes) < 1.1 * len(pickle.dumps(ta))
    b = back[0]
    b.propagate_until(1.0)
    assert np.array_equal(np.asarray(b.state), np.asarray(ret[-1][0].state))
    ta.propagate_until(1.0)  # (an integrator that has propagated carries its bookkeeping)
    assert len(pickle.dumps(ret[0][0])) < 1.1 * len(pickle.dumps(ta))
    # a result is its own: writing to one leaves the others
    other = np.asarray(ret[1][0].state).copy()
    ret[0][0].state[:] = 7.0
    assert np.array_equal(np.asarray(ret[1][0].state), other)
