"""CPU test of the donation ring's counters: warps that wait past their bound close the ring and leave,
and no item is lost."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_waiting_threads_leave_a_closed_ring_without_losing_items(tmp_path):
    exe = str(tmp_path / "ring_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-o", exe,
                    os.path.join(ROOT, "tests", "native", "ring_test.cpp"), "-I",
                    os.path.join(ROOT, "gcsm-bu_b200", "csrc")], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.startswith("ok"), p.stdout + p.stderr
