"""Transposed and complex solves of chains whose vectors leave room for one CTA per
SM run level after level in a workspace of the call's own: the dataflow sweeps'
bits (one instance), also from two streams at once and from a captured graph,
which runs the sweeps."""
import numpy as np
import pytest
import torch

from neospice_b200.solver import Batch, Topology, _interleave

pytestmark = pytest.mark.gpu

N, COUNT = 9800, 149


def _chain(complex_):
    rng = np.random.default_rng([98, complex_])
    k = np.arange(N - 1)
    rows, cols = np.r_[np.arange(N), k, k + 1], np.r_[np.arange(N), k + 1, k]
    v = np.r_[6.0 + rng.random(N), rng.uniform(-1, 1, 2 * N - 2)]
    if complex_:
        v = v + 1j * np.r_[np.zeros(N), rng.uniform(-1, 1, 2 * N - 2)]
    at = np.lexsort((rows, cols))
    cp = np.searchsorted(cols[at], np.arange(N + 1)).astype(np.int32)
    return N, cp, rows[at].astype(np.int32), v[at]


@pytest.mark.parametrize("complex_", [False, True])
def test_levels_equal_sweeps(complex_):
    m = _chain(complex_)
    topo = Topology.order_complex(*m) if complex_ else Topology.order(*m)
    rhs = np.random.default_rng(99).uniform(-1, 1, (2, N * (2 if complex_ else 1)))
    solve, want = None, None
    for count in (1, COUNT):
        batch = Batch([topo] * count)
        v = torch.from_numpy(np.tile(_interleave(m[3]), count)).cuda()
        if complex_:
            lu, st = batch.refactor_complex(v)
            solve = lambda x, b=batch, f=lu: b.solve_complex(f, x)  # noqa: E731
        else:
            st, _ = batch.refactor(v)
            solve = batch.solve_transposed
        assert int(st.abs().sum()) == 0
        x = [torch.from_numpy(np.tile(r, count)).cuda() for r in rhs]
        torch.cuda.synchronize()
        if count == 1:
            want = [solve(y) for y in x]
            continue
        streams = [torch.cuda.Stream() for _ in x]
        got = []
        for s, y in zip(streams, x):
            with torch.cuda.stream(s):
                got.append([y.clone() for _ in range(4)])
        for k in range(4):  # both streams' solves in flight together
            for s, y in zip(streams, got):
                with torch.cuda.stream(s):
                    solve(y[k])
        torch.cuda.synchronize()
        for y, w in zip(got, want):
            for z in y:
                assert torch.equal(z.view(count, -1), w.expand(count, -1))
        z = x[0].clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            solve(z)
        z.copy_(x[0])
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(z.view(count, -1), want[0].expand(count, -1))
