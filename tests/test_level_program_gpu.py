"""Level programs on the GPU: operating points of linear circuits below the
AMD-LU threshold are one factorization and one solve of the first matrix, so
DcBatch must give the oracle's refactor + solve bit for bit.  Sizes around a
warp and around the program's bound on updates per unknown (sparse trees have
a program at every size, resistor meshes only up to a side of about ten)."""
import numpy as np
import pytest

import oracle
from neospice_b200 import workloads as W
from neospice_b200.circuit import GND, Circuit, DcBatch
from neospice_b200.solver import Topology

pytestmark = pytest.mark.gpu


def _mesh(rng, side):
    c = Circuit(side * side)
    grid = np.arange(side * side, dtype=np.int32).reshape(side, side)
    for a, b in ((grid[:, :-1].ravel(), grid[:, 1:].ravel()), (grid[:-1].ravel(), grid[1:].ravel())):
        c.add_resistors(a, b, np.exp(0.3 * rng.standard_normal(len(a))))
    c.I(GND, side * side - 1, 1e-3)
    c.V(0, GND, 1.0)
    return c.finalize()


def _tree(rng, nodes):
    return W.resistor_network(rng, nodes).build()


@pytest.mark.parametrize("make,sizes", [(_tree, [1, 2, 30, 31, 32, 33, 127, 128, 254]),
                                        (_mesh, [2, 3, 6, 9, 10, 11, 12, 15])])
def test_linear_operating_points_match_oracle(make, sizes):
    circuits = [make(np.random.default_rng([71, s]), s) for s in sizes]
    sols, status, _ = (batch := DcBatch(circuits, symbolic=DcBatch.PER_INSTANCE)).run()
    assert int(status.abs().sum()) == 0
    for s, c, x in zip(sizes, circuits, batch.split(sols)):
        cp, ri = c.pattern()
        a, rhs = c.initial_matrix(1e-12)
        st = oracle.Structure(len(cp) - 1, *Topology.order(len(cp) - 1, cp, ri, a).export())
        rc, lu, _ = oracle.port_refactor(st, a)
        assert rc == 0
        np.testing.assert_array_equal(x, oracle.port_solve(st, lu, rhs), err_msg=str(s))
