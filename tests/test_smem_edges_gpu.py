"""Batches whose shared memory lies just below the 48 KB a launch may use without
asking: the kernels' static shared memory counts too, so the largest sizes below
it need the larger limit set as well.  Chains of the orders at which the sweeps
(12 bytes an unknown) and the refactors (a column buffer per warp and 4 bytes an
unknown) reach 48 KB, for one instance; A x against b row by row."""
import numpy as np
import pytest
import torch

from neospice_b200.solver import Batch, Topology, _interleave

pytestmark = pytest.mark.gpu


def _chain(n, complex_=False):
    """Tridiagonal CSC (n, col_ptr, row_idx, values), diagonally dominant."""
    rng = np.random.default_rng([85, n])
    k = np.arange(n - 1)
    rows, cols = np.r_[np.arange(n), k, k + 1], np.r_[np.arange(n), k + 1, k]
    v = np.r_[6.0 + rng.random(n), rng.uniform(-1, 1, 2 * n - 2)]
    if complex_:
        v = v + 1j * np.r_[np.zeros(n), rng.uniform(-1, 1, 2 * n - 2)]
    at = np.lexsort((rows, cols))
    cp = np.searchsorted(cols[at], np.arange(n + 1)).astype(np.int32)
    return n, cp, rows[at].astype(np.int32), v[at]


def _check(m, x, b, transposed=False):
    n, cp, ri, v = m
    cols = np.repeat(np.arange(n), np.diff(cp))
    r, c = (cols, ri) if transposed else (ri, cols)
    y = np.zeros(n, v.dtype)
    np.add.at(y, r, v * x[c])
    # pivots of at least 3, |x| below 1 and some ten roundings of terms below 9
    np.testing.assert_allclose(y, b, rtol=0, atol=100 * np.finfo(float).eps)


@pytest.mark.parametrize("n", [4010, 4011, 4093, 4095, 4096, 4097, 11262, 11263, 11264])
def test_real(n):
    m = _chain(n)
    batch = Batch([Topology.order(*m)])
    st, _ = batch.refactor(torch.from_numpy(m[3]).cuda())
    assert int(st[0]) == 0
    b = np.random.default_rng(86).uniform(-1, 1, n)
    _check(m, batch.solve(torch.from_numpy(b).cuda()).cpu().numpy(), b)
    _check(m, batch.solve_transposed(torch.from_numpy(b).cuda()).cpu().numpy(), b, True)


@pytest.mark.parametrize("n", [2406, 2407, 2455, 2456, 2457, 2458, 10238, 10239, 10240])
def test_complex(n):
    m = _chain(n, complex_=True)
    batch = Batch([Topology.order_complex(*m)])
    lu, st = batch.refactor_complex(torch.from_numpy(_interleave(m[3])).cuda())
    assert int(st[0]) == 0
    b = np.random.default_rng(87).uniform(-1, 1, n) + 0j
    x = batch.solve_complex(lu, torch.from_numpy(_interleave(b)).cuda()).cpu().numpy()
    _check(m, x[0::2] + 1j * x[1::2], b)
