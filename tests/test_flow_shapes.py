"""The launch functions of a batch's refactors and solves against stand-ins for the
CUDA runtime (tests/cpp/flow_shape_check.cpp, linked here with the library's
own objects): the shape follows what fits an SM, not the instance count alone.  And
which plans are solved with a thread per row."""
import pathlib
import subprocess

from neospice_b200 import build as nb

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_flow_shapes(tmp_path):
    objs = [nb._obj(nb.CSRC / "kernels" / k) for k in ("lu_kernels.cu", "lu_complex.cu")]
    if not all(o.exists() for o in objs):
        nb.build()
    exe = tmp_path / "flow_shape_check"
    subprocess.run([nb.nvcc(), *nb.COMMON, str(ROOT / "tests" / "cpp" / "flow_shape_check.cpp"),
                    *map(str, objs), "-o", str(exe), "-cudart", "shared", "-lcudart",
                    f"-I{nb.CSRC}"], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "0 failure(s)" in res.stdout
