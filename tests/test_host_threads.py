"""Batch creation where the system grants fewer threads than asked for: the work runs
on those there are, and nothing aborts the process."""
import pathlib
import shutil
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]

SCRIPT = """
import resource
import numpy as np
from neospice_b200 import _lib as L, workloads as W
from neospice_b200.circuit import DcBatch, TranBatch
circuits = [W.resistor_network(np.random.default_rng([88, k]), 20).build() for k in range(24)]
pages = int(open("/proc/self/statm").read().split()[0])
size = pages * resource.getpagesize() + (20 << 20)  # two threads' stacks of 8 MiB
resource.setrlimit(resource.RLIMIT_AS, (size, size))
try:
    if {tran}:
        TranBatch(circuits, 1e-12, 1e-10, np.zeros(1, np.int32))
    else:
        DcBatch(circuits, symbolic=DcBatch.PER_INSTANCE)
except L.NsgError as e:
    print(e)
print("returned")
"""


@pytest.mark.parametrize("tran", [False, True])
def test_batch_create_without_threads(tran):
    res = subprocess.run([sys.executable, "-c", SCRIPT.format(tran=tran)], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, (res.returncode, res.stderr[-500:])
    assert "returned" in res.stdout and "unavailable" not in res.stdout, res.stdout


def test_on_threads(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "threads_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", f"-I{ROOT / 'neospice_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "threads_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "0 failure(s)" in res.stdout, res.stdout + res.stderr
