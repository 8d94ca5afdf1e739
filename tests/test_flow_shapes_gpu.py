"""The launch shapes of a batch's dataflow kernels give one instance's bits: 297
instances (four CTAs of 8 warps per SM, or two of 16 where fewer than needed fit)
against one (a CTA of 16 warps), real and complex, at the orders where the shape
changes and beside dense blocks."""
import numpy as np
import pytest
import torch

from neospice_b200.solver import Batch, Topology, _interleave

pytestmark = pytest.mark.gpu


def _matrix(n, dense, seed):
    """A chain whose last `dense` unknowns are coupled with one another."""
    rng = np.random.default_rng([91, seed])
    k = np.arange(n - 1)
    r, c = np.meshgrid(np.arange(n - dense, n), np.arange(n - dense, n))
    at = np.unique(np.concatenate([np.arange(n) * (n + 1), k * n + k + 1, (k + 1) * n + k,
                                   (c * n + r).ravel()]).astype(np.int64))
    cols, rows = at // n, at % n
    v = rng.uniform(-1, 1, len(at)) + 1j * rng.uniform(-1, 1, len(at))
    v[rows == cols] += 3.0 * (dense + 2)
    cp = np.searchsorted(cols, np.arange(n + 1)).astype(np.int32)
    return n, cp, rows.astype(np.int32), v


# complex vectors fit four times up to 2816 unknowns, real ones three times up to 6314;
# 150 coupled unknowns leave no room for six complex column buffers
@pytest.mark.parametrize("n,dense", [(1, 1), (33, 33), (300, 2), (500, 150), (2816, 40),
                                     (2817, 40), (6314, 60), (6315, 60)])
def test_many_equal_one(n, dense):
    m = _matrix(n, dense, n)
    rng = np.random.default_rng([92, n])
    b = rng.standard_normal(n) * (rng.random(n) < 0.7)
    out = []
    for count in (1, 297):
        real = Batch([Topology.order(m[0], m[1], m[2], m[3].real.copy())] * count)
        st, _ = real.refactor(torch.from_numpy(np.tile(m[3].real, count)).cuda())
        assert int(st.abs().sum()) == 0
        x = torch.from_numpy(np.tile(b, count)).cuda()
        size = topo_nlu(real)
        got = [real.lu_values().reshape(count, -1)[:, :size],
               real.solve(x.clone()).cpu().numpy().reshape(count, -1),
               real.solve_transposed(x.clone()).cpu().numpy().reshape(count, -1)]
        cplx = Batch([Topology.order_complex(*m)] * count)
        lu, st = cplx.refactor_complex(torch.from_numpy(np.tile(_interleave(m[3]), count)).cuda())
        assert int(st.abs().sum()) == 0
        x = torch.from_numpy(np.tile(_interleave(b + 1j * b[::-1]), count)).cuda()
        got += [lu.cpu().numpy().reshape(count, -1)[:, :2 * topo_nlu(cplx)],
                cplx.solve_complex(lu, x).cpu().numpy().reshape(count, -1)]
        out.append(got)
    for one, many in zip(*out):
        np.testing.assert_array_equal(many, np.broadcast_to(one, many.shape))


def topo_nlu(batch):
    return batch.topologies[0].info()["nnz_lu"]
