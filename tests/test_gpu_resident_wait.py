"""A resident pass that loses a message between two blocks ends by itself with a status, and the plan is
usable afterwards (tests/resident_wait.cu)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(engine, tmp_path_factory):
    from rtmuq2d_gb300 import build
    build.build()
    exe = str(tmp_path_factory.mktemp("wait") / "resident_wait")
    objs = [os.path.join(build.OUT, s + ".o") for s in ("rtm_kernels.cu", "rtm_resident.cu", "rtm_host.c", "rtm_zfp.c")]
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + [os.path.join(ROOT, "tests", "resident_wait.cu")] + objs +
                   ["-o", exe], check=True)
    return exe


# one, two and more columns a thread (the last with its values in tensor memory), and double
@pytest.mark.parametrize("grid", ((96, 64, 16, 0, 1), (901, 301, 40, 0, 2), (1201, 403, 40, 0, 4), (150, 90, 20, 1, 1),
                                  (1000, 300, 40, 1, 2)))
def test_lost_message_ends_the_pass(program, grid):
    r = subprocess.run([program] + [str(v) for v in grid], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
