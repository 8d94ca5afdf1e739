"""The dataflow complex refactor and sweeps against the general kernels, bit for
bit: the same batch with a factor array that is 16-byte aligned (dataflow) and
one that is not (general), at the edges of runs and warps and for both launch
shapes; and the solutions against numpy."""
import numpy as np
import pytest
import torch

from neospice_b200.solver import Batch, Topology, _interleave

pytestmark = pytest.mark.gpu


def _matrix(n, dense, seed):
    rng = np.random.default_rng([76, seed])
    m = np.zeros((n, n), complex)
    k = np.arange(n - 1)
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    m[k, k + 1], m[k + 1, k] = z(n - 1), z(n - 1)
    m[n - dense:, n - dense:] = z(dense, dense)
    m[np.arange(n), np.arange(n)] = 4.0 + 2 * n + z(n)
    cols, rows = np.nonzero(m.T)
    cp = np.searchsorted(cols, np.arange(n + 1)).astype(np.int32)
    return m, n, cp, rows.astype(np.int32), m.T[cols, rows]


SHAPES = [(1, 1), (2, 2), (14, 3), (17, 5), (30, 9), (40, 32), (60, 33), (90, 66), (200, 38)]


@pytest.mark.parametrize("count", [len(SHAPES), 160])
def test_dataflow_equals_general(count):
    mats = [_matrix(n, d, k) for k, (n, d) in enumerate(SHAPES)]
    topos = [Topology.order_complex(*m[1:]) for m in mats]
    pick = [k % len(mats) for k in range(count)]
    batch = Batch([topos[k] for k in pick])
    ax = torch.from_numpy(np.concatenate([_interleave(mats[k][4]) for k in pick])).cuda()
    rng = np.random.default_rng(77)
    rhs = [rng.standard_normal(mats[k][1]) * (rng.random(mats[k][1]) < 0.7) + 0j for k in pick]
    b = torch.from_numpy(np.concatenate([_interleave(r) for r in rhs])).cuda()
    size = 2 * int(batch.lu_offsets[-1])
    out = []
    for shift in (0, 1):
        lu = torch.zeros(size + 1, dtype=torch.float64, device="cuda")[shift:shift + size]
        lu, st = batch.refactor_complex(ax, d_lu=lu)
        assert int(st.abs().sum()) == 0
        out.append((lu, batch.solve_complex(lu, b.clone())))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])
    x = out[0][1].cpu().numpy()
    for i, k in enumerate(pick[:len(mats)]):
        n = mats[k][1]
        at = 2 * int(batch.vector_offsets[i])
        # diagonally dominant by a factor near 2: a few n ulp of the rhs
        np.testing.assert_allclose(mats[k][0] @ (x[at:at + 2 * n:2] + 1j * x[at + 1:at + 2 * n:2]),
                                   rhs[i], rtol=0, atol=100 * n * np.finfo(float).eps * 4)
