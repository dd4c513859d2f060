"""The lane form's warps meet at a CTA barrier every few iterations: lanes that
need very different numbers of steps, CTAs with a few threads and with threads
that return early, and lanes taken from the queue all give the oracle's bits."""

import numpy as np
import pytest

import hyk
from hyk import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["persistent", "plain", "plain_inplace"])
@pytest.mark.parametrize("form", ["lane", "global"])
@pytest.mark.parametrize("n", [1, 37, 257, 40000])
def test_uneven_step_counts_bitwise(oracle, n, form, mode):
    if n == 40000 and mode != "persistent":
        n = 1300
    sys_ = W.kepler_sys()
    st = W.kepler_ics(n, seed=13)
    # from one step to some forty, in runs of lanes so that whole warps finish early
    tf = np.where(np.arange(n) % 97 < 70, 0.01, np.random.default_rng(n).uniform(0.5, 6.0, n))
    kw = {"global_jets": True} if form == "global" else {}
    ta = hyk.taylor_adaptive_batch(sys_, st, tol=1e-15, team_size=1, prop_mode=mode, **kw)
    ta.propagate_until(tf)
    o = oracle.Oracle(sys_, st, order=ta.order, mode=1)
    r = o.propagate_until(tf)
    assert np.array_equal(np.asarray(ta.state), o.state)
    assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy(), r["n_steps"].astype(np.int64))
