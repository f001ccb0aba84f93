"""The run lists of the FP64 and FP32 steps against the general pull and class
rules, and the cover of the FP16 form's tiles, on the CPU: native/run_lists.cu over the smallest boxes, the test cases' and random
ones (openings next to the inlets, rows shorter and longer than a warp)."""
import os
import random
import subprocess

import pytest

from tests.cases import GOLDEN_CASES, ORACLE_CASES
from tmixer_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    build.build()
    out = str(tmp_path_factory.mktemp("native") / "run_lists")
    cmd = [build._nvcc(), "-O1", "-std=c++17"] + build.ARCH + ["-o", out, os.path.join(HERE, "native", "run_lists.cu"),
                                                              build.LIB, "-Xlinker", "-rpath=" + build.PKG]
    subprocess.run(cmd, check=True)
    return out


def _cases():
    keys = ("inx", "iny", "nz", "mnx", "mny", "ia")
    out = [[5, 3, 3, 3, 3, 2], [12, 4, 520, 4, 5, 4], [401, 51, 51, 101, 750, 151][:6], [8, 3, 3, 3, 3, 5]]
    out += [[c[k] for k in keys] for c in [v[0] for v in GOLDEN_CASES.values()] + list(ORACLE_CASES.values())]
    rng = random.Random(7)
    for _ in range(60):
        mnx = rng.randint(3, 70)
        inx = mnx + 2 + rng.randint(0, 80)
        out.append([inx, rng.randint(3, 12), rng.randint(3, 9), mnx, rng.randint(3, 20), rng.randint(2, inx - mnx)])
    return out


def test_run_lists(checker):
    args = [str(v) for c in _cases() for v in c]
    r = subprocess.run([checker] + args, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
