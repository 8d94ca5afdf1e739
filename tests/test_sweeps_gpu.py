"""Row sweeps at the edges of their chunks: rows of up to 31, 32, 33, 64, 65 and
130 entries (dense trailing blocks of those orders behind a sparse chain), more
rows than one pass of a CTA's warps takes (512 and its neighbours), one row
alone, and AMD-LU plans; bit for bit against the oracle's solve."""
import numpy as np
import pytest
import torch

import oracle
from neospice_b200.solver import Batch, Topology

pytestmark = pytest.mark.gpu


def _matrix(n, dense, seed):
    """A chain of n unknowns whose last `dense` are fully coupled."""
    rng = np.random.default_rng([73, seed])
    m = np.zeros((n, n))
    k = np.arange(n - 1)
    m[k, k + 1], m[k + 1, k] = rng.standard_normal(n - 1), rng.standard_normal(n - 1)
    m[n - dense:, n - dense:] = rng.standard_normal((dense, dense))
    m[np.arange(n), np.arange(n)] = 4.0 + n + rng.random(n)
    cols, rows = np.nonzero(m.T)
    cp = np.searchsorted(cols, np.arange(n + 1)).astype(np.int32)
    return n, cp, rows.astype(np.int32), m.T[cols, rows]


SIZES = [(1, 1), (2, 2), (40, 32), (60, 33), (100, 34), (90, 64), (300, 66), (511, 2), (512, 1),
         (513, 131), (1100, 5)]


@pytest.mark.parametrize("solver", ["markowitz", "amdlu"])
def test_row_sweeps_match_oracle(solver):
    mats = [_matrix(n, d, k) for k, (n, d) in enumerate(SIZES)]
    topos = [Topology.order(*m, solver=solver) for m in mats]
    batch = Batch(topos)
    st, _ = batch.refactor(torch.from_numpy(np.concatenate([m[3] for m in mats])).cuda())
    assert int(st.abs().sum()) == 0
    rng = np.random.default_rng(74)
    rhs = [np.where(rng.random(m[0]) < 0.3, 0.0, rng.standard_normal(m[0])) for m in mats]
    x = batch.solve(torch.from_numpy(np.concatenate(rhs)).cuda()).cpu().numpy()
    xt = batch.solve_transposed(torch.from_numpy(np.concatenate(rhs)).cuda()).cpu().numpy()
    lu = batch.lu_values()
    for k, (m, t) in enumerate(zip(mats, topos)):
        at = slice(batch.vector_offsets[k], batch.vector_offsets[k + 1])
        if solver == "amdlu":
            dense = np.zeros((m[0], m[0]))
            dense[m[2], np.repeat(np.arange(m[0]), np.diff(m[1]))] = m[3]
            # strongly diagonally dominant (condition below 10): a few n ulp
            tol = 50 * m[0] * np.finfo(float).eps * np.abs(rhs[k]).max()
            np.testing.assert_allclose(dense @ x[at], rhs[k], rtol=0, atol=tol)
            np.testing.assert_allclose(dense.T @ xt[at], rhs[k], rtol=0, atol=tol)
            continue
        s = oracle.Structure(m[0], *t.export())
        f = lu[batch.lu_offsets[k]:batch.lu_offsets[k] + s.n_elem]
        np.testing.assert_array_equal(x[at], oracle.port_solve(s, f, rhs[k]))
        np.testing.assert_array_equal(xt[at], oracle.port_solve(s, f, rhs[k], transposed=True))
