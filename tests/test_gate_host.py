"""The order of cooperative launches, on the CPU (tests/gate_check.cc)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launches_that_may_run_together_fit_the_sms(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "gate_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "rtmuq2d_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "gate_check.cc"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
