"""Trees whose levels are wide enough are solved with a thread per row and a barrier per
level: bit for bit the general kernels' results, which run the same batch
level after level in global memory (a schedule, a chain too long for shared
memory beside it, or a factor array that is not 16-byte aligned), on both sides
of the rule's line."""
import numpy as np
import pytest
import torch

from neospice_b200.solver import Batch, Topology, _interleave

pytestmark = pytest.mark.gpu


def _tree(n, spread, seed):
    """Node k hangs from one of the `spread` nodes before it."""
    rng = np.random.default_rng([93, seed])
    k = np.arange(1, n)
    p = np.array([int(rng.integers(max(0, j - spread), j)) for j in k], int)
    rows, cols = np.r_[np.arange(n), k, p], np.r_[np.arange(n), p, k]
    z = rng.uniform(-1, 1, 2 * (n - 1)) + 1j * rng.uniform(-1, 1, 2 * (n - 1))
    v = np.r_[np.full(n, 3.0) + 3 * np.bincount(np.r_[k, p], minlength=n), z]
    at = np.lexsort((rows, cols))
    cp = np.searchsorted(cols[at], np.arange(n + 1)).astype(np.int32)
    return n, cp, rows[at].astype(np.int32), v[at]


def _wide(topo):
    i = topo.info()
    return 8 * (i["nnz_lu"] - i["n"]) * i["fwd_levels"] <= i["n"] ** 2


SIZES = [(1, 1), (33, 33), (300, 300), (600, 600), (5000, 5000), (3000, 20), (40, 1)]


@pytest.mark.parametrize("engine", ["markowitz", "auto-amdlu"])
def test_real(engine):
    mats = [_tree(n, s, k) for k, (n, s) in enumerate(SIZES)]
    topos = [Topology.order(m[0], m[1], m[2], m[3].real.copy(), solver=engine) for m in mats]
    assert {_wide(t) for t in topos} == {True, False}
    chain = _tree(17100, 1, 99)  # 12 bytes an unknown: more than a CTA may have
    long = Topology.order(chain[0], chain[1], chain[2], chain[3].real.copy())
    rng = np.random.default_rng(94)
    b = np.concatenate([rng.standard_normal(m[0]) * (rng.random(m[0]) < 0.7) for m in mats])
    values = np.concatenate([m[3].real for m in mats])
    out = []
    for extra in (False, True):
        batch = Batch(topos + [long] * extra)
        v = torch.from_numpy(np.r_[values, chain[3].real] if extra else values).cuda()
        x = torch.from_numpy(np.r_[b, np.ones(chain[0])] if extra else b).cuda()
        if extra:
            batch.set_schedule(1)
        st, _ = batch.refactor(v)
        assert int(st.abs().sum()) == 0
        out.append([f(x.clone()).cpu().numpy()[:len(b)]
                    for f in (batch.solve, batch.solve_transposed)])
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("count", [1, 150, 297])
def test_complex(count):
    mats = [_tree(n, s, k) for k, (n, s) in enumerate(SIZES)]
    topos = [Topology.order_complex(*m) for m in mats]
    pick = [k % len(mats) for k in range(count + len(mats) - 1)]
    batch = Batch([topos[k] for k in pick])
    ax = torch.from_numpy(np.concatenate([_interleave(mats[k][3]) for k in pick])).cuda()
    rng = np.random.default_rng(95)
    b = torch.from_numpy(rng.standard_normal(2 * sum(mats[k][0] for k in pick))).cuda()
    size = 2 * int(batch.lu_offsets[-1])
    out = []
    for shift in (0, 1):
        lu = torch.zeros(size + 1, dtype=torch.float64, device="cuda")[shift:shift + size]
        lu, st = batch.refactor_complex(ax, d_lu=lu)
        assert int(st.abs().sum()) == 0
        out.append(batch.solve_complex(lu, b.clone()))
    assert torch.equal(out[0], out[1])
