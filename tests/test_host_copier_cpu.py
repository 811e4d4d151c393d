"""Host threads of the large copies: tests/host_copier_check.cpp is built
against the library's cf1_hostcopier.h and copies with all threads, with fewer
and with none to be had.  Whole numbers: equality."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cf1_rs_b200", "csrc")


def test_copies_with_fewer_threads(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("needs g++")
    exe = str(tmp_path / "host_copier_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", os.path.join(HERE, "host_copier_check.cpp"),
                    "-o", exe, "-ldl"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
