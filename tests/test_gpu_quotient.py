"""The division of the resident PCG's scalars (quotient in csrc/flof_common.cuh)
against the FP64 division (tests/quotient.cu)."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_quotient_rounds_the_division(gpu, tmp_path):
    from ofblend_gb300 import build

    exe = str(tmp_path / "quotient")
    subprocess.run([build.nvcc()] + build.flags() + [os.path.join(ROOT, "tests", "quotient.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    print(r.stdout)
