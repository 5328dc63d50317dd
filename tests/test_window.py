"""CPU test of the window search that the enumeration kernel uses on sorted lists."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_window_search_over_all_list_sizes(tmp_path):
    exe = str(tmp_path / "window_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-o", exe, os.path.join(ROOT, "tests", "native", "window_test.cpp"),
                    "-I", os.path.join(ROOT, "gcsm-bu_b200", "csrc")], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.startswith("ok"), p.stdout + p.stderr
