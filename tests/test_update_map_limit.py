"""Circuit batches whose plans have no update map (nsg_set_update_map_limit) are
refused with an error, also where the circuit is small and sparse enough for a
level program.  Each case runs in a process of its own: the limit is
process-wide."""
import pathlib
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]

SCRIPT = """
import numpy as np
from neospice_b200 import _lib as L, workloads as W
from neospice_b200.circuit import DcBatch, TranBatch
assert L.lib().nsg_set_update_map_limit(0) == L.NSG_OK
circuits = [W.inverter_chain_mc(np.random.default_rng(3), 32).build(),
            W.resistor_network(np.random.default_rng(4), 60).build()]
try:
    if {tran}:
        TranBatch(circuits, 1e-12, 1e-10, np.zeros(1, np.int32))
    else:
        DcBatch(circuits, symbolic=DcBatch.PER_INSTANCE)
except L.NsgError as e:
    print(e)
"""


@pytest.mark.parametrize("tran", [False, True])
def test_batch_without_update_map_is_refused(tran):
    res = subprocess.run([sys.executable, "-c", SCRIPT.format(tran=tran)], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, (res.returncode, res.stderr[-500:])
    assert "no update map" in res.stdout, res.stdout
