"""GPU test of a batch that runs out of host memory half way (native program, its own operator new[])."""
import os
import shutil
import subprocess

import pytest

import csm

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_batch_out_of_host_memory_is_not_half_applied(tmp_path):
    lib = os.path.dirname(csm.LIB_PATH)
    exe = str(tmp_path / "host_oom")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-o", exe, os.path.join(ROOT, "tests", "native", "host_oom.cpp"),
                    "-L", lib, "-lcsm", f"-Wl,-rpath,{lib}"], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.startswith("ok"), p.stdout + p.stderr
