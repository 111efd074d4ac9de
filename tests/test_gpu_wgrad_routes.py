"""Weight gradients of the warm-start network's stride-1 layers at extents where
the rule takes halo tiles and where it takes im2col (tests/wgrad_routes.cu)."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_weight_gradients_of_both_forms(gpu, tmp_path):
    from ofblend_gb300 import build

    exe = str(tmp_path / "wgrad_routes")
    src = [os.path.join(ROOT, "tests", "wgrad_routes.cu")]
    src += [os.path.join(build.CSRC, f) for f in ("flof_conv_tc.cu", "flof_ops.cu")]
    subprocess.run([build.nvcc()] + build.flags() + src + ["-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    print(r.stdout)
