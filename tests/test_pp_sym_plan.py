"""The plan of the pair-once sum on the host: no heap memory, whole ranges."""
import os
import subprocess

from conftest import ROOT


COUNTING = """
#include <cstdlib>
#include <new>
int allocations = 0;
void *operator new(size_t bytes) { ++allocations; return std::malloc(bytes); }
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }
"""


def test_plan(tmp_path):
    from nbody_gb300 import build

    counting = tmp_path / "counting.cpp"
    counting.write_text(COUNTING)

    exe = str(tmp_path / "plan")
    subprocess.run([build.NVCC] + build.FLAGS + [os.path.join(ROOT, "tests", "pp_sym_plan_check.cu"), str(counting),
                    "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
