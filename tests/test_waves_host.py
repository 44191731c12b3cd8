"""A server's choice of the resident members that run at a step, on the CPU (tests/waves_check.cc)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_member_falls_behind(tmp_path):
    gxx = shutil.which("g++")
    inc = next((d for d in ("/usr/local/cuda/include", os.environ.get("CUDA_HOME", "") + "/include")
                if os.path.exists(os.path.join(d, "cuda_runtime.h"))), None)
    if gxx is None or inc is None:
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path / "waves_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", inc, "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "rtmuq2d_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "waves_check.cc"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
