"""What a differentiable propagation holds until its backward pass: the rows
of its tape that were filled, not the room it was taken with."""

import numpy as np
import pytest
import torch

import hyk
from hyk import workloads as W
from hyk.adjoint import taylor_flow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,t", [(1, 0.0), (3, 0.5), (16384, 20.0)])
def test_tape_keeps_the_filled_rows(n, t):
    st, mu = W.cr3bp_ics(n, seed=3)
    x0 = torch.tensor(st, device="cuda", requires_grad=True)
    pars = torch.tensor(mu, device="cuda", requires_grad=True)
    x, _ = taylor_flow(W.cr3bp_sys(), x0, t, pars=pars, tol=1e-15)
    rows = max(1, int(x.grad_fn.saved_tensors[3].max()))
    for v, width in zip(x.grad_fn.saved_tensors[:3], (6, 1, 1)):
        assert v.shape[0] == rows and v.untyped_storage().nbytes() == rows * width * n * 8
    gx, gp = torch.autograd.grad(x, (x0, pars), torch.ones_like(x))
    assert torch.isfinite(gx).all() and torch.isfinite(gp).all()
    if t == 0.0:
        assert torch.equal(gx, torch.ones_like(gx)) and not gp.any()


def test_segments_hold_their_own_rows():
    """Four segments in one graph take about as much as one propagation of their length."""
    st = W.pendulum_ics(20000, seed=1)

    def held(k):
        torch.cuda.empty_cache()
        base = torch.cuda.memory_allocated()
        x = torch.tensor(st, device="cuda", requires_grad=True)
        y = x
        for _ in range(k):
            y, _ = taylor_flow(W.pendulum_sys(), y, 4.0 / k)
        used = torch.cuda.memory_allocated() - base
        (g,) = torch.autograd.grad(y, x, torch.ones_like(y))
        assert torch.isfinite(g).all()
        return used

    held(1)  # (modules)
    one, four = held(1), held(4)
    assert four < 1.5 * one + 20000 * 8 * 100


def test_gradient_does_not_depend_on_the_room(monkeypatch):
    import hyk.adjoint as A

    st = W.kepler_ics(77, seed=5)
    tf = torch.tensor(np.random.default_rng(1).uniform(0.1, 3.0, 77), device="cuda")
    out = []
    for cap in (1, 7, 1024):
        monkeypatch.setattr(A, "_tape_cap", lambda ne, B, c=cap: c)
        x0 = torch.tensor(st, device="cuda", requires_grad=True)
        x, _ = taylor_flow(W.kepler_sys(), x0, tf)
        out.append((x.detach(), torch.autograd.grad(x, x0, torch.ones_like(x))[0]))
    for x, g in out[1:]:
        assert torch.equal(x, out[0][0]) and torch.equal(g, out[0][1])
