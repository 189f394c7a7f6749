"""The direct sum's scratch where device memory is short: the pair-once form falls
back once, keeps what is there, and later calls neither wait nor allocate (a host
program over a device memory with a budget)."""
import os
import subprocess

from conftest import ROOT


def test_scratch_where_memory_is_short(tmp_path):
    from nbody_gb300 import build

    exe = str(tmp_path / "scratch_check")
    subprocess.run([build.NVCC, "-O1", "-std=c++17", "-x", "cu", "-I", build.CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "scratch_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
