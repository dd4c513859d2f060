"""Single precision outside the register form: as many CTAs on an SM as the
shared memory holds, the registers that the global-memory grid leaves, and
batch sizes around the places where the placement changes, with the oracle's bits."""

import numpy as np
import pytest
import torch

import hyk
from hyk import cos, exp, log, sin, sqrt

pytestmark = pytest.mark.gpu


def functions(k):
    """k coupled copies of six equations with elementary functions."""
    v = hyk.make_vars(*["m{}".format(i) for i in range(6 * k)])
    out = []
    for j in range(k):
        a, b, c, d, e, f = v[6 * j:6 * j + 6]
        z = v[(6 * j + 7) % (6 * k)]
        out += [(a, sin(b) * exp(-c)), (b, a / (1.0 + d * d)), (c, sqrt(1.0 + a * a) - c), (d, cos(e) - d * f),
                (e, log(2.0 + f * f) * 0.3), (f, -a * b + e - 0.1 * z)]
    return out


def chain(n):
    v = hyk.make_vars(*["l{}".format(i) for i in range(n)])
    return [(v[i], v[i] * (1.0 - v[i] - 0.1 * v[(i + 1) % n] * v[(i + 2) % n])) for i in range(n)]


@pytest.mark.parametrize("name", ["functions", "chain"])
def test_registers_let_the_ctas_in(name):
    sys_ = functions(1) if name == "functions" else chain(4)
    ta = hyk.taylor_adaptive_batch(sys_, np.ones((len(sys_), 8), np.float32), team_size=1, fp_type=np.float32)
    assert ta.module_info["smem_per_lane"] > 0 and ta.module_info["ctas_per_sm"] == 2


@pytest.mark.parametrize("name", ["shared", "global"])
@pytest.mark.parametrize("k", range(7))
def test_batch_sizes_bitwise(oracle, name, k):
    subs = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    n = [1, 31, 33, subs + 1, 32 * subs, 32 * subs + 1, 64 * subs + 45][k]
    sys_ = functions(1 if name == "shared" else 3)
    st = np.random.default_rng(k).uniform(0.5, 1.0, (len(sys_), n)).astype(np.float32)
    tf = np.random.default_rng(7).uniform(0.1, 0.8, n).astype(np.float32)
    pick = np.unique(np.linspace(0, n - 1, 64).astype(np.int64))
    for mode in ("persistent", "plain_inplace"):
        ta = hyk.taylor_adaptive_batch(sys_, st, team_size=1, fp_type=np.float32, prop_mode=mode)
        assert (ta.module_info["smem_per_lane"] == 0) == (name == "global")
        ta.propagate_until(tf)
        o = oracle.Oracle(sys_, np.ascontiguousarray(st[:, pick]).astype(np.float64), order=ta.order, mode=1, prec=2)
        r = o.propagate_until(tf[pick].astype(np.float64))
        assert np.array_equal(np.asarray(ta.state)[:, pick].astype(np.float64), o.state)
        assert np.array_equal(ta.propagate_res_tensors["n_steps"].cpu().numpy()[pick], r["n_steps"].astype(np.int64))
