"""Forms at the limit of the shared memory: the one chosen for a batch can be
built when a system's team layout fits only with cold state rows, asked for
without them; and a team whose layout fits only without the slots of its
powers' spread products does without those."""

import ctypes

import numpy as np
import pytest
import torch

import hyk
from hyk import _lib
from hyk.core import _form_for
from hyk.decompose import taylor_decompose

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 64, 3000, 100000])
@pytest.mark.parametrize("bodies,order", [(10, 100), (6, 60)])
@pytest.mark.parametrize("flags", [0, _lib.HYK_CFG_NO_COLD_ROWS])
def test_team_fits_the_shared_memory(libhyk, flags, bodies, order, n):
    dec = taylor_decompose(hyk.model.nbody(bodies))
    team, out = _form_for(dec, order, 0, flags, n)
    assert flags & out == flags
    if team <= 1:
        return
    d, keep = dec.as_c()
    fits = []
    for f in {out, out | _lib.HYK_CFG_NO_COLD_ROWS}:
        cfg, ns = _lib.hyk_config_t(32, 0, f, team), ctypes.c_uint32()
        assert libhyk.hyk_codegen_check(ctypes.byref(d), order, ctypes.byref(cfg), 2, None, 0, ctypes.byref(ns), None) == 0
        fits.append(32 // team * ns.value * 8 <= torch.cuda.get_device_properties(0).shared_memory_per_block_optin)
    assert any(fits)


def _powers(n):
    v = hyk.make_vars(*["x{}".format(i) for i in range(n)])
    rhs = [-0.1 * v[i] * v[(i + 1) % n] for i in range(n)]
    for i in range(16):
        rhs[i] = rhs[i] + 0.01 * (1.0 + v[i] * v[(i + 3) % n]) ** (-1.5 if i < 8 else -0.5)
    return list(zip(v, rhs))


@pytest.mark.parametrize("cold_rows", [True, False])
@pytest.mark.parametrize("n", [118, 120, 124])  # 29055, 29465, 30285 slots with the products' 1584; 29056 fit
def test_team_whose_spread_products_do_not_fit(oracle, n, cold_rows):
    sys_, st = _powers(n), np.random.default_rng(n).uniform(0.5, 1.5, (n, 5))
    ta = hyk.taylor_adaptive_batch(sys_, st, tol=1e-86, team_size=32, cold_rows=cold_rows)
    assert ta.order == 101 and ta.module_info["team_size"] == 32
    o = oracle.Oracle(sys_, st, order=101, mode=1)
    for _ in range(2):
        ta.step()
        o.step()
    assert np.array_equal(np.asarray(ta.state), o.state)
