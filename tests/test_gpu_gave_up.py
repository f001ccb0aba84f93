"""The flag that a step sets when its copies did not arrive: every read and every
timing reports it, and a whole new state (init, restore, the first mixer of an
empty batch) clears it.  The flag is host memory, which the test writes itself: a
handle takes the first free one of a page.  And the wait itself, in a kernel of its
own."""
import ctypes
import os
import subprocess

import pytest

import tmixer_b200 as T
from tests.cases import GOLDEN_CASES, to_spec
from tmixer_b200 import build

pytestmark = pytest.mark.gpu


def _next_flag():
    """The flag that the next handle or batch will take."""
    take, give = T.lib()["_ZN8tmx_host15error_flag_takeEv"], T.lib()["_ZN8tmx_host15error_flag_giveEPi"]
    take.restype, take.argtypes = ctypes.POINTER(ctypes.c_int), []
    give.restype, give.argtypes = None, [ctypes.POINTER(ctypes.c_int)]
    f = take()
    give(f)
    return f


def _raises(call):
    with pytest.raises(T.TmxError, match="gave up waiting"):
        call()


@pytest.mark.parametrize("precision", [T.TMX_FP64, T.TMX_FP32])
def test_solver(gpu, precision):
    spec = to_spec(GOLDEN_CASES["tiny_ref"][0])
    spec.precision = precision
    flag = _next_flag()
    with T.Solver(spec) as s:
        s.init().step(3)
        ck = s.checkpoint()
        flag[0] = 1
        for call in (s.sync, s.sums, s.mixing, s.checkpoint, lambda: s.field(0, "rho"), lambda: s.step_timed(2),
                     lambda: s.time_steps(2)):
            _raises(call)
        s.restore(ck).step(2)
        s.sync()
        flag[0] = 1
        _raises(s.sync)
        s.init().step(2)
        assert s.step_timed(1)[2] > 0


@pytest.mark.parametrize("precision", [T.TMX_FP64, T.TMX_FP32])
def test_batch(gpu, precision):
    spec = to_spec(GOLDEN_CASES["tiny_ref"][0])
    spec.precision = precision
    flag = _next_flag()
    with T.Batch(precision, budget=4 * T.Batch.footprint(spec)) as B:
        a, b = B.add(spec), B.add(spec)
        B.step(3)
        flag[0] = 1
        for call in (B.sync, B.outlet_im, B.health, lambda: B.field(a, 0, "rho"), lambda: B.checkpoint(a),
                     lambda: B.step_timed(2), lambda: B.time_steps(2), lambda: B.tune(2)):
            _raises(call)
        B.remove(a)
        c = B.add(spec)  # (b's state is still the one that the flag is about)
        _raises(B.sync)
        B.remove(b)
        B.remove(c)
        B.add(spec)
        B.step(2)
        B.sync()
        assert B.time_steps(2) > 0


def test_wait_runs_out(gpu, tmp_path):
    out = str(tmp_path / "give_up")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "give_up.cu")
    subprocess.run([build._nvcc(), "-O1", "-std=c++17"] + build.ARCH + ["-o", out, src], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
