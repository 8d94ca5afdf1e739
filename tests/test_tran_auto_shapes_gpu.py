"""The launch shapes that transient batches choose by themselves give the results of the
shapes that can be asked for, bit for bit: CTAs of 256 threads for up to one
instance per SM, of 128 or 256 for more (256 where a family has more than 128
devices), of 512, one or two per SM, above 128 unknowns."""
import numpy as np
import pytest

from neospice_b200 import workloads as W
from neospice_b200.circuit import TranBatch

pytestmark = pytest.mark.gpu

PULSE = (0.0, 1.8, 0.0, 1e-11, 1e-11, 1e-9, 2e-9)


def _results(netlists, shape):
    b = TranBatch([n.build() for n in netlists], 1e-12, 1.5e-11, np.arange(3, dtype=np.int32),
                  max_points=400)
    b.set_shape(*shape)
    b.run()
    return b.results()


# stages, instances, shapes asked for (64 stages: 128 MOSFETs, 65: 130; 128
# stages: 130 unknowns)
@pytest.mark.parametrize("stages,count,asked", [
    (8, 1, [(512, 2), (256, 4), (128, 8)]),      # chosen: 256 threads, one per SM
    (64, 149, [(512, 2), (256, 4), (128, 8)]),   # 128, four
    (65, 149, [(512, 2), (256, 4)]),             # 256, two
    (128, 1, [(512, 2)]),                        # 512, one
    (128, 149, [(512, 2)]),                      # 512, two
])
def test_chosen_equal_asked(stages, count, asked):
    netlists = [W.inverter_chain_mc(np.random.default_rng([96, k]), stages, pulse=PULSE)
                for k in range(count)]
    chosen = _results(netlists, (0, 0))
    assert all(r["status"] == 0 for r in chosen)
    for shape in asked:
        for r, s in zip(chosen, _results(netlists, shape)):
            np.testing.assert_array_equal(s["time"], r["time"])
            np.testing.assert_array_equal(s["values"], r["values"])
            assert s["newton_iters"] == r["newton_iters"]
