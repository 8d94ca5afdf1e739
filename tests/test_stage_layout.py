"""The span of an instance's workspace that a launch stages in shared memory holds
nothing that no kernel reads (tests/cpp/stage_check.cpp, linked here with the
library)."""
import pathlib
import subprocess

from neospice_b200 import build as nb

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_stage_layout(tmp_path):
    lib = nb.build()
    exe = tmp_path / "stage_check"
    subprocess.run([nb.nvcc(), *nb.COMMON, str(ROOT / "tests" / "cpp" / "stage_check.cpp"),
                    "-o", str(exe), str(lib), "-Xlinker", f"-rpath={lib.parent}"], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "0 failure(s)" in res.stdout, res.stdout + res.stderr
