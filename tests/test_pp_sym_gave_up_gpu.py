"""A pair-once sum that is not whole writes nothing: the kernel's own range check
(no fault, no wait) makes one CTA give up."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_sum_that_is_not_whole_writes_nothing(cuda, tmp_path):
    from nbody_gb300 import build

    exe = str(tmp_path / "gave_up")
    subprocess.run([build.NVCC] + build.FLAGS + [os.path.join(ROOT, "tests", "pp_sym_gave_up_check.cu"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
