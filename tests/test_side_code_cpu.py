"""Side-set codes on the host: tests/side_code_check.cpp is built against the
library's cf1_common.cuh and compares the code every k-mer occurrence carries
through phase 3 with the side-set byte of the general rule, over all
neighbours and over self loops.  Whole numbers: equality."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cf1_rs_b200", "csrc")


def test_side_codes_match_the_side_set_bytes(tmp_path):
    cxx = shutil.which("g++")
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not cxx or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA runtime headers")
    exe = str(tmp_path / "side_code_check")
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{inc}", f"-I{CSRC}", os.path.join(HERE, "side_code_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
