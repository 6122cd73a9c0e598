"""Scratch buffers that grow in a shared pool (tests/cpp/scratch_check.cc, on
the CPU): a buffer's old range is released only after the work queued on it is
done, and a stream of equal blocks keeps the buffers of its first block (all
but a few in a hundred streams, whose merge sets fall another way)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_growing_scratch(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "scratch_check")
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I",
                        os.path.join(ROOT, "libfalcon_dsp_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "scratch_check.cc"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "400"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    ok, streams, blocks, grew = r.stdout.split()
    assert ok == "ok" and int(streams) > 350 and int(blocks) > 10 * int(streams) // 2
    assert int(grew) <= int(streams) // 20
