"""The form chosen for a batch can be built: a system whose team layout fits
the shared memory only with cold state rows, asked for without them."""

import ctypes

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
