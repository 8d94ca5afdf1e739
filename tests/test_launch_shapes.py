"""The Newton kernels' launch functions against stand-ins for the CUDA runtime
(tests/cpp/launch_check.cpp, linked here with the library's own objects)."""
import pathlib
import subprocess

from neospice_b200 import build as nb

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_launch_shapes(tmp_path):
    objs = [nb._obj(nb.CSRC / "kernels" / k) for k in ("transient.cu", "newton_dc.cu")]
    if not all(o.exists() for o in objs):
        nb.build()
    host = [str(nb.CSRC / "host" / f) for f in ("amd_lu.cpp", "plan.cpp", "sparse_order.cpp")]
    exe = tmp_path / "launch_check"
    subprocess.run([nb.nvcc(), *nb.COMMON, str(ROOT / "tests" / "cpp" / "launch_check.cpp"), *host,
                    *map(str, objs), "-o", str(exe), "-cudart", "shared", "-lcudart",
                    f"-I{nb.CSRC}"], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "0 failure(s)" in res.stdout
