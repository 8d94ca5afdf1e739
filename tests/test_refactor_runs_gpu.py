"""The run-wise refactor at the edges of its runs and groups: dense trailing
blocks of 1 to 10 and of 33 to 69 columns (runs of every length modulo 4, common
rows around one and two warps) behind a chain and behind scattered columns, and
more metadata than one window of 32 entries; factors bit for bit against the
oracle's, for numeric() and refactorize()."""
import numpy as np
import pytest
import torch

import oracle
from neospice_b200.solver import Batch, Topology

pytestmark = pytest.mark.gpu


def _matrix(n, dense, scattered, seed):
    rng = np.random.default_rng([75, seed])
    m = np.zeros((n, n))
    k = np.arange(n - 1)
    m[k, k + 1], m[k + 1, k] = rng.standard_normal(n - 1), rng.standard_normal(n - 1)
    m[n - dense:, n - dense:] = rng.standard_normal((dense, dense))
    for i, j in rng.integers(0, n, (scattered, 2)):
        m[i, j] = rng.standard_normal()
    m[np.arange(n), np.arange(n)] = 4.0 + n + rng.random(n)
    cols, rows = np.nonzero(m.T)
    cp = np.searchsorted(cols, np.arange(n + 1)).astype(np.int32)
    return n, cp, rows.astype(np.int32), m.T[cols, rows]


@pytest.mark.parametrize("count", [1, 200, 320])
@pytest.mark.parametrize("check", [False, True])
def test_runs_match_oracle(count, check):
    shapes = [(d + 12, d, 0) for d in (*range(1, 11), 33, 36, 37, 65, 69)]
    shapes += [(150, 20, 200), (90, 1, 60), (300, 40, 300)]
    mats = [_matrix(n, d, s, k) for k, (n, d, s) in enumerate(shapes)]
    topos = [Topology.order(*m) for m in mats]
    pick = [k % len(mats) for k in range(max(count, len(mats) if count > 1 else 1))]
    if count == 1:
        pick = [len(mats) - 1]
    batch = Batch([topos[k] for k in pick])
    a = torch.from_numpy(np.concatenate([mats[k][3] for k in pick])).cuda()
    st, _ = batch.refactor(a, check_pivots=check)
    assert int(st.abs().sum()) == 0
    lu = batch.lu_values()
    want = {}
    for i, k in enumerate(pick):
        if k not in want:
            s = oracle.Structure(mats[k][0], *topos[k].export())
            rc, f, _ = oracle.port_refactor(s, mats[k][3])
            assert rc == 0
            want[k] = f
        at = batch.lu_offsets[i]
        np.testing.assert_array_equal(lu[at:at + len(want[k])], want[k])
