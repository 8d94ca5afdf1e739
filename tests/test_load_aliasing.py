"""The device loads declare their pointers as not overlapping: no host call passes
one array for two of them (tests/cpp/load_alias_check.cpp)."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
CSRC = ROOT / "neospice_b200" / "csrc"


def test_host_loads_do_not_alias(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "load_alias_check"
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{CSRC}",
                    str(ROOT / "tests" / "cpp" / "load_alias_check.cpp"),
                    str(CSRC / "host" / "mos1_card.cpp"), str(CSRC / "host" / "bsim4_card.cpp"),
                    "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and " 0 failure(s)" in res.stdout, res.stdout + res.stderr
