"""The wait of the FP64 and FP32 steps for their copies runs out: a kernel of its own
whose copies never come."""
import os
import subprocess

import pytest

from tmixer_b200 import build

pytestmark = pytest.mark.gpu


def test_wait_runs_out(gpu, tmp_path):
    out = str(tmp_path / "give_up")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "give_up.cu")
    subprocess.run([build._nvcc(), "-O1", "-std=c++17"] + build.ARCH + ["-o", out, src], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
