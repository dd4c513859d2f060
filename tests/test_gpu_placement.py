"""The placement of trajectories on the resident warps: at batch sizes around
the places where it changes (one unit per warp, a full warp on every
sub-partition, a quarter more, beyond every resident warp) every form and
propagation kernel gives every trajectory the oracle's bits, and the reverse
sweep the bits it has in a batch of a few lanes."""

import numpy as np
import pytest
import torch

import hyk
from hyk import workloads as W
from hyk.adjoint import taylor_flow

pytestmark = pytest.mark.gpu

FORMS = {
    "lane": {},
    "global": {"global_jets": True, "team_size": 1},
    "team": {"team_size": 16},
}


def sizes(form, n_sm):
    subs = 4 * n_sm  # sub-partitions: one warp each in the first layers
    full = subs * (2 if form == "team" else 32)
    return [1, subs - 1, subs + 1, full, full + 1, full + full // 4, full + full // 4 + 1, 2 * full + 45]


@pytest.mark.parametrize("k", range(8))
@pytest.mark.parametrize("form", list(FORMS))
def test_batch_sizes_bitwise(oracle, form, k):
    n = sizes(form, torch.cuda.get_device_properties(0).multi_processor_count)[k]
    sys_ = W.pendulum_sys()
    st = W.pendulum_ics(n, seed=71 + k)
    tf = np.random.default_rng(k).uniform(0.05, 0.9, n)
    for mode in ("persistent", "plain", "plain_inplace"):
        ta = hyk.taylor_adaptive_batch(sys_, st, tol=2.2e-16, prop_mode=mode, **FORMS[form])
        ta.step()
        o = oracle.Oracle(sys_, st, order=ta.order, mode=1)
        o.step()
        assert np.array_equal(np.asarray(ta.state), o.state), mode
        ta.propagate_until(1.0 + tf)
        r = o.propagate_until(1.0 + tf)
        assert np.array_equal(np.asarray(ta.state), o.state), mode
        assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy(), r["n_steps"].astype(np.int64)), mode


@pytest.mark.parametrize("k", range(1, 8))
def test_reverse_sweep_batch_sizes_bitwise(k):
    n = sizes("global", torch.cuda.get_device_properties(0).multi_processor_count)[k]
    st = W.pendulum_ics(n, seed=91)
    tf = torch.tensor(np.random.default_rng(9).uniform(0.05, 0.9, n), device="cuda")
    x0 = torch.tensor(st, device="cuda", requires_grad=True)
    x, _ = taylor_flow(W.pendulum_sys(), x0, tf)
    (g,) = torch.autograd.grad(x, x0, torch.ones_like(x))
    pick = np.unique(np.linspace(0, n - 1, 37).astype(np.int64))
    y0 = x0.detach()[:, pick].contiguous().requires_grad_(True)
    y, _ = taylor_flow(W.pendulum_sys(), y0, tf[pick])
    (gy,) = torch.autograd.grad(y, y0, torch.ones_like(y))
    assert torch.equal(x.detach()[:, pick], y.detach()) and torch.equal(g[:, pick], gy)
