"""Solves do not depend on the wait limit.  After a good refactor every batched
solve (real, transposed, complex, grid-wide) whose dependency waits give up at
once (nsg_set_wait_limit(0)) must still return the values of the default limit
bit for bit: the calls report no status, so a wait that gives up may not show."""
import numpy as np
import pytest
import torch

from matrices import banded
from neospice_b200 import _lib as L
from neospice_b200 import workloads as W
from neospice_b200.solver import Batch, Topology, _interleave

pytestmark = pytest.mark.gpu


def _with_limit(polls, call):
    assert L.lib().nsg_set_wait_limit(polls) == L.NSG_OK, L.lib().nsg_last_error()
    try:
        x = call()
        torch.cuda.synchronize()
        return x
    finally:
        assert L.lib().nsg_set_wait_limit(L.NSG_DEFAULT_WAIT_LIMIT) == L.NSG_OK


def _matrices():
    c = W.diode_mesh(np.random.default_rng(81), side=20).build()
    cp, ri = c.pattern()
    return [banded(1500, 7, seed=82), (len(cp) - 1, cp, ri, c.initial_matrix(1e-12)[0])]


@pytest.mark.parametrize("schedule", [0, 2])
@pytest.mark.parametrize("solver", ["markowitz", "amdlu"])
def test_real_solves(solver, schedule):
    mats = _matrices() if solver == "markowitz" else \
        [_matrices()[0], W.power_grid_transient(40)]
    batch = Batch([Topology.order(*m, solver=solver) for m in mats])
    batch.set_schedule(schedule)
    st, _ = batch.refactor(torch.from_numpy(np.concatenate([m[3] for m in mats])).cuda())
    assert int(st.abs().sum()) == 0
    n = int(batch.vector_offsets[-1])
    b = torch.from_numpy(np.random.default_rng(83).standard_normal(n)).cuda()
    for solve in (batch.solve, batch.solve_transposed):
        want = solve(b.clone())
        torch.cuda.synchronize()
        assert torch.isfinite(want).all()
        assert torch.equal(_with_limit(0, lambda: solve(b.clone())), want)


def test_complex_solve():
    n, cp, ri, v = _matrices()[1]
    rng = np.random.default_rng(84)
    z = v + 1j * 1e-3 * rng.standard_normal(len(v))
    batch = Batch([Topology.order_complex(n, cp, ri, z)] * 3)
    lu, st = batch.refactor_complex(torch.from_numpy(np.tile(_interleave(z), 3)).cuda())
    assert int(st.abs().sum()) == 0
    b = torch.from_numpy(rng.standard_normal(6 * n)).cuda()
    want = batch.solve_complex(lu, b.clone())
    torch.cuda.synchronize()
    assert torch.isfinite(want).all()
    assert torch.equal(_with_limit(0, lambda: batch.solve_complex(lu, b.clone())), want)
