"""The form chosen for a batch: teams where they spread a small batch over the
GPU, the lane form where the batch fills it and the lane form is the faster one
there, but teams throughout for a system whose lane form spills."""

import pytest
import torch

import hyk
from hyk import var
from hyk import workloads as W
from hyk.core import _form_for
from hyk.decompose import taylor_decompose

pytestmark = pytest.mark.gpu


def _ring(n):
    v = hyk.make_vars(*["l{}".format(i) for i in range(n)])
    return [(v[i], v[(i + 1) % n] * 0.9 - v[(i - 1) % n] * 1.1) for i in range(n)]


SYSTEMS = {
    "bodies": lambda: hyk.model.nbody(4, Gconst=1.0, masses=[1.0, 0.1, 0.05, 0.02]),
    "ring": lambda: _ring(9),
    "variational": lambda: var.var_ode_sys(W.kepler_sys(), var.var_args.vars, order=1).sys,
}


# lanes per sub-partition, and whether teams are the faster form there
@pytest.mark.parametrize("name,lanes,teams", [
    ("bodies", 1, True), ("bodies", 20, True), ("bodies", 100, False), ("bodies", 400, False), ("bodies", 1600, False),
    ("ring", 1, True), ("ring", 16, True), ("ring", 48, False), ("ring", 400, False),
    ("variational", 5, True), ("variational", 50, True), ("variational", 100, True), ("variational", 400, True),
])
def test_form_of_full_batches(libhyk, name, lanes, teams):
    subs = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    team, _ = _form_for(taylor_decompose(SYSTEMS[name]()), 20, 0, 0, lanes * subs)
    assert (team > 1) == teams
