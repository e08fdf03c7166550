"""The z transforms' rows lie inside one warp and exchange through shared memory between warp barriers.
The kernels' source, run on the host one lane after the other (zrow_lanes.cpp), gives the right
transforms in any order of the lanes between the barriers."""
import pathlib
import shutil
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent
ROOT = HERE.parent
CUDA = pathlib.Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent

# a transform of N <= 512 Gaussian values and back: a few dozen roundings of values of order 1 to 5
TOL = {"f32": 1e-5, "f64": 2e-14}


def test_rows_do_not_depend_on_the_order_of_the_lanes(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not (CUDA / "include" / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path / "zrow_lanes"
    subprocess.run([gxx, "-std=c++17", "-O1", "-w", f"-I{ROOT / 'include'}", f"-I{ROOT / 'lucky_droplets_b200' / 'csrc'}",
                    f"-I{CUDA / 'include'}", str(HERE / "zrow_lanes.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [line.split() for line in out if line]
    assert len(rows) == 40  # ten lengths, two precisions, two orders
    bad = [r for r in rows if not float(r[3]) < TOL[r[0]]]
    assert not bad, bad
