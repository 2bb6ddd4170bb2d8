"""The library's host code where the device says no: run without a GPU, in a
child process whose CUDA runtime calls go to a stand-in (fake_cudart.cpp) that
refuses or delays what a test asks it to and counts the kernels launched."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = "/usr/local/cuda/include"

PRELUDE = """
import ctypes, os, sys, threading, time
sys.path.insert(0, {here!r}); sys.path.insert(0, os.path.dirname({here!r}))
import numpy as np
import fomo_julia_b200 as F
from cases import layered
from test_gpu_routes import OpenShot
fake = ctypes.CDLL(None)
fake.fake_get.restype = ctypes.c_long
fake.fake_set.argtypes = [ctypes.c_char_p, ctypes.c_long]
def get(k): return fake.fake_get(k.encode())
def put(k, v): fake.fake_set(k.encode(), v)
b = F.backend("b200")
case = lambda nx=150, nz=90, **kw: layered(nx, nz, seed=4, **dict(dict(nbc=12, fd_order=8, nt=600), **kw))
SPLIT = "13stress_kernel"
MARCH = "12march_kernel"
"""


@pytest.fixture(scope="session")
def host_run(tmp_path_factory):
    """Runs a script against the stand-in runtime."""
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE):
        pytest.skip("needs g++ and the CUDA headers")
    from fomo_julia_b200 import build
    build.build()
    so = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CUDA_INCLUDE,
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", str(so), "-lpthread"], check=True)

    def run(script, **env):
        e = {k: v for k, v in os.environ.items() if not k.startswith("FOMO_B200_")}
        e.update(LD_PRELOAD=str(so), PYTHONDONTWRITEBYTECODE="1", **env)
        r = subprocess.run([sys.executable, "-c", PRELUDE.format(here=HERE) + script], capture_output=True, text=True,
                           env=e, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return run


def test_the_stand_in_runs_a_shot(host_run):
    host_run("""
s = OpenShot(case(), b)
s.advance(600)
assert s.k.value == 600 and s.finish()[2] == 3          # 256 steps a launch
assert get("launches:resident_kernel") == 3 and get("launches:" + SPLIT) == 0
""")


@pytest.mark.parametrize("after", [0, 1])
def test_refused_cooperative_launch_runs_the_split_launches(host_run, after):
    host_run(f"""
put("refuse_cooperative_after", {after})
s = OpenShot(case(), b)
s.advance(600)
assert s.k.value == 600
assert get("launches:resident_kernel") == {after}
assert get("launches:" + SPLIT) == 600 - 256 * {after}
s.finish()
""")


def test_no_room_for_the_mailboxes_runs_the_split_launches(host_run):
    host_run("""
s = OpenShot(case(), b)
F.set_step_kernel("split")
s.advance(1)                                              # everything but the mailboxes is allocated
F.set_step_kernel("auto")
put("fail_alloc_max", 1 << 40); put("fail_alloc_min", 0)
for _ in range(3):
    s.advance(100)
assert s.k.value == 301
assert get("launches:resident_kernel") == 0 and get("launches:" + SPLIT) == 301
assert get("failed_allocs") == 2                          # one attempt a shot, and its retry after a trim
s.finish()
""")


def test_mailboxes_are_given_back_when_memory_runs_short(host_run):
    host_run("""
s = OpenShot(case(), b)
s.advance(100)
held = get("live_bytes")
put("capacity", get("reserved"))
try:
    F.Wavefield(400, 400, b)
except F._lib.FomoError as e:
    assert "FOMO_ENOMEM" in str(e)
else:
    raise AssertionError("allocated beyond the capacity")
assert get("live_bytes") < held
put("capacity", 1 << 36)
s.advance(500)                                            # allocated again
assert s.k.value == 600 and get("launches:" + SPLIT) == 0
s.finish()
""")
