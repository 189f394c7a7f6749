"""The links of the child table on the host: whole trees, and trees whose prefix
sums or keys are broken as a wait that ran out would leave them (no GPU runs on
one of those)."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from nbody_gb300 import build

    exe = str(tmp_path_factory.mktemp("tree_links") / "tree_links_check")
    subprocess.run([build.NVCC, "-O1", "-std=c++17", "-x", "cu", "-I", build.CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "tree_links_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("bodies,systems,bits", [(2, 1, 63), (3, 1, 2), (9, 1, 63), (1000, 1, 63), (5000, 1, 9),
                                                 (5000, 1, 30), (20011, 1, 63), (5000, 3, 63), (20011, 40, 12)])
def test_links(check, bodies, systems, bits):
    r = subprocess.run([check, str(bodies), str(systems), str(bits), "1"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
