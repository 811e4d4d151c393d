"""The kernels' word-wise byte copy on the host: tests/byte_copy_check.cpp is
built against the library's cf1_common.cuh and carries the copy out over all
alignments of both ends and lengths 0..64.  Whole numbers: equality."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cf1_rs_b200", "csrc")


def test_byte_copy_stays_inside_the_source(tmp_path):
    cxx = shutil.which("g++")
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not cxx or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA runtime headers")
    exe = str(tmp_path / "byte_copy_check")
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{inc}", f"-I{CSRC}", os.path.join(HERE, "byte_copy_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
