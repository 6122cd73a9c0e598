"""How the tensor-core planner's slots are stored, on random channel sets
(tests/cpp/tc_store_check.cc over the library's own planner)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tc_store_flags(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "tc_store_check")
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I",
                        os.path.join(ROOT, "libfalcon_dsp_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "tc_store_check.cc"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "2000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
