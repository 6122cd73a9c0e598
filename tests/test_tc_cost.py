"""The tensor-core launch's item list and its cut by cost for calls whose cost
does not fit 32 bits, and for ordinary ones (tests/cpp/tc_cost_check.cc over
the library's own planner): every item in exactly one CTA's run."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAX_N = 2 ** 31 - 1


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("tc_cost") / "tc_cost_check")
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I",
                        os.path.join(ROOT, "libfalcon_dsp_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "tc_cost_check.cc"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


# channels, decimation, taps a phase, up, samples; whether the work is past 2^32 units
@pytest.mark.parametrize("nch,d,taps,up,n,past", [
    (32, 10, 4095, 1, MAX_N, True),
    (64, 16, 4000, 1, MAX_N, True),
    (256, 32, 2048, 1, MAX_N, True),
    (1, 1, 16383, 1, MAX_N, True),
    (1, 1, 24000, 1, 1 << 30, True),
    (8, 1, 4095, 1, 1 << 30, True),
    (5, 7, 1000, 3, MAX_N, False),
    (64, 16, 4000, 1, 1 << 30, False),
    (1, 10, 4095, 1, 1 << 24, False),
    (3, 5, 60, 2, 70_001, False),
])
def test_items_are_partitioned(check, nch, d, taps, up, n, past):
    r = subprocess.run([check, str(nch), str(d), str(taps), str(up), str(n)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    ok, items, unit, work = r.stdout.split()
    assert ok == "ok" and (int(work) >= 1 << 32) == past
    assert (int(unit) > 0) == (int(work) >= 1 << 31)
