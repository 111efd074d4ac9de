"""Contexts on several devices of one process share no budget of SMs and no
kernel attribute (csrc/flof_device.h), checked on the host."""
import os
import subprocess

from conftest import ROOT


def test_state_is_kept_per_device(tmp_path):
    exe = str(tmp_path / "per_device")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "ofblend_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "per_device.cc"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
