"""The lane form's CTA barrier with lanes that stop before the recurrences of
an iteration: a batch or an ensemble's group in which a state becomes
non-finite, and a tape that fills, with the oracle's bits."""

import numpy as np
import pytest
import torch

import hyk
from hyk import workloads as W
from hyk.adjoint import _propagate_taped
from hyk.core import get_module

pytestmark = pytest.mark.gpu

FORMS = {"lane": {}, "global": {"global_jets": True}}


def _ics(n, bad, speed):
    """Kepler orbits; the lanes bad are slowed or sped up to where their state overflows."""
    st = W.kepler_ics(n, seed=31)
    st[3:, bad] *= speed
    return st


@pytest.mark.parametrize("mode", ["persistent", "plain"])
@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("n,bad", [(300, [5]), (1000, [0, 999]), (42000, [17]), (42000, [41990])])
def test_batch_with_a_non_finite_lane(oracle, n, bad, form, mode):
    sys_, st = W.kepler_sys(), _ics(n, bad, 1e10)  # overflow after 32 steps or so
    tf = np.random.default_rng(n).uniform(0.05, 20.0, n)
    tf[bad] = 1e300
    ta = hyk.taylor_adaptive_batch(sys_, st, tol=1e-15, team_size=1, prop_mode=mode, **FORMS[form])
    ta.propagate_until(tf)
    o = oracle.Oracle(sys_, st, order=ta.order, mode=1)
    r = o.propagate_until(tf)
    oc = ta.propagate_res_tensors["outcome"].cpu().numpy()
    assert (oc[bad] == int(hyk.taylor_outcome.err_nf_state)).any()
    assert np.array_equal(oc, r["outcome"].astype(np.int64))
    assert np.array_equal(np.asarray(ta.state), o.state, equal_nan=True)
    assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy(), r["n_steps"].astype(np.int64))


@pytest.mark.parametrize("batch", [1, 4, 12])
@pytest.mark.parametrize("form", list(FORMS))
def test_ensemble_with_a_non_finite_iteration(oracle, form, batch):
    """Several groups to a warp, one of which stops."""
    sys_, n_iter = W.kepler_sys(), 50
    st = _ics(n_iter * batch, [7 * batch], 0.0)  # a fall into the centre: 223 steps
    ta = hyk.taylor_adaptive_batch(sys_, np.ascontiguousarray(st[:, :batch]), tol=1e-15, team_size=1, **FORMS[form])

    def gen(t, i):
        t.state[:] = np.ascontiguousarray(st[:, i * batch:(i + 1) * batch])
        return t

    ret = hyk.ensemble_propagate_until(ta, 60.0, n_iter, gen, max_steps=400)
    for i in range(0, n_iter, 7):
        o = oracle.Oracle(sys_, np.ascontiguousarray(st[:, i * batch:(i + 1) * batch]), order=ta.order, mode=1)
        o.propagate_until(60.0, max_steps=400)
        assert np.array_equal(np.asarray(ret[i][0].state), o.state, equal_nan=True), i


@pytest.mark.parametrize("cap", [1, 3, 6])
@pytest.mark.parametrize("form", list(FORMS))
def test_tape_that_fills(form, cap):
    """More lanes than slots, uneven step counts, a tape grown several times."""
    n = 42000
    st = W.kepler_ics(n, seed=33)
    tf = np.random.default_rng(2).uniform(0.05, 4.0, n)
    ta = hyk.taylor_adaptive_batch(W.kepler_sys(), st, tol=1e-15, team_size=1, **FORMS[form])
    mod = get_module(ta._dec, ta.order, 0, team_size=1, **FORMS[form])
    x, th, a, ck_x, ck_t, ck_h = _propagate_taped(mod, torch.tensor(st, device="cuda"), None,
                                                  torch.zeros(n, dtype=torch.float64, device="cuda"),
                                                  torch.tensor(tf, device="cuda"), cap=cap)
    ta.propagate_until(tf)
    assert np.array_equal(x.cpu().numpy(), np.asarray(ta.state)) and torch.equal(th, ta._thi)
    assert torch.equal(a["n_iter"], ta.propagate_res_tensors["n_iter"]) and int(a["n_iter"].max()) > cap
    assert torch.equal(ck_x[0], torch.tensor(st, device="cuda"))
    # the last step of every lane ends at its final state's time
    k = (a["n_iter"] - 1).unsqueeze(0)
    assert np.allclose((ck_t.gather(0, k) + ck_h.gather(0, k))[0].cpu().numpy(), tf, rtol=1e-14)
