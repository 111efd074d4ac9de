"""The chained PCG's predicted beta against freshly summed z.r (tests/cg_beta.cu
on the kernels of csrc/flof_solve.cu)."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_predicted_beta(gpu, tmp_path):
    from ofblend_gb300 import build

    exe = str(tmp_path / "cg_beta")
    src = [os.path.join(ROOT, "tests", "cg_beta.cu")]
    src += [os.path.join(build.CSRC, f) for f in ("flof_solve.cu", "flof_ops.cu")]
    subprocess.run([build.nvcc()] + build.flags() + src + ["-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
