"""The rule that keeps a body point's 13×13 window inside the finest grid
(window_inside, ibpm.jl_b200/csrc/ibpm_internal.cuh), by which a problem refuses
its body points and a step clamps moved ones: on the CPU, at the first and last
index of both directions, beyond the range of an int (where an index saturates
and idx + 6 wraps), at infinities and at no number."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ibpm.jl_b200", "csrc")
NX, NY = 64, 32
OUTSIDE = ["6", "0", "-1", "2147483641", "2147483642", "2147483647", "2147483648", "-2147483648", "1e300", "-1e300", "inf",
           "-inf", "nan"]


def test_window_inside(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "window_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC,
                    os.path.join(ROOT, "tests", "window_check.cu"), "-o", exe], check=True)
    cases = [((x, y), True) for x in ("7", str(NX - 6)) for y in ("7", str(NY - 6))]
    cases += [((x, "16"), False) for x in OUTSIDE + [str(NX - 5)]]
    cases += [(("16", y), False) for y in OUTSIDE + [str(NY - 5)]]
    out = subprocess.run([exe, str(NX), str(NY), *[v for p, _ in cases for v in p]], check=True, capture_output=True,
                         text=True, timeout=60).stdout.strip()
    assert [c == "1" for c in out] == [inside for _, inside in cases]
