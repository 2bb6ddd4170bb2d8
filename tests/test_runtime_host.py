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
def steps(): return get("launches:" + SPLIT) + get("launches:" + MARCH)  # of the split launches and the fused step
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
                           env=e, timeout=60)
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
def test_refused_cooperative_launch_runs_other_launches(host_run, after):
    host_run(f"""
put("refuse_cooperative_after", {after})
s = OpenShot(case(), b)
s.advance(600)
assert s.k.value == 600
assert get("launches:resident_kernel") == {after}
assert steps() == 600 - 256 * {after}
s.finish()
""")


def test_no_room_for_the_mailboxes_runs_other_launches(host_run):
    host_run("""
s = OpenShot(case(), b)
F.set_step_kernel("split")
s.advance(1)                                              # everything but the mailboxes is allocated
F.set_step_kernel("auto")
put("fail_alloc_max", 1 << 40); put("fail_alloc_min", 0)
for _ in range(3):
    s.advance(100)
assert s.k.value == 301
assert get("launches:resident_kernel") == 0 and steps() == 301
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
assert s.k.value == 600 and steps() == 0
s.finish()
""")


def test_single_shots_beside_served_ones_share_the_device(host_run):
    host_run("""
c = case()
s = OpenShot(c, b)
H = F.init_habc(s.med.nx, s.med.nz, c.nbc, c.dt, c.dx, c.dz, c.v_ref, b)
a, par = F.get_fd_coefficients(8), F.sim_params(c.dt, c.nt, c.dx, c.dz, 8)
src, rec = F.Source(60, 30, F.ricker_wavelet(c.f0, c.dt, c.nt)), F.setup_receivers(c.rec_x, c.rec_z, s.med)
with F.ShotServer() as srv:
    put("hold", 1)
    t = srv.submit(s.med, H, a, src, rec, par)
    bad = F.Source(10 ** 6, 30, src.wavelet)
    try:
        srv.submit(s.med, H, a, bad, rec, par)            # refused: not in flight
    except F._lib.FomoError:
        pass
    t0 = time.time()
    s.advance(40)                                         # the served shot is in flight: launches of 32 steps
    assert get("launches:resident_kernel") == 2
    put("launch_us", 20000)
    s.advance(70)                                         # three launches, the first two with pauses of twice their time
    assert get("launches:resident_kernel") == 5 and time.time() - t0 > 2 * 0.04 + 3 * 0.02
    put("launch_us", 0)
    put("hold", 0)
    srv.wait(t, timeout=60)
    s.advance(490)                                        # alone again: 256 steps a launch
    assert s.k.value == 600 and get("launches:resident_kernel") == 7
    put("hold", 1)
    more = [srv.submit(s.med, H, a, src, rec, par) for _ in range(3)]
    put("hold", 0)
    srv.wait_all(more, timeout=60)
    s2 = OpenShot(c, b)
    s2.advance(600)
    assert get("launches:resident_kernel") == 10 and get("launches:" + SPLIT) == 0
""")


SERVED = """
c = case(nt=40, n_rec=5)
med = F.init_medium(c.vp, c.vs, c.rho, c.dx, c.dz, c.nbc, 8, b)
H = F.init_habc(med.nx, med.nz, c.nbc, c.dt, c.dx, c.dz, c.v_ref, b)
a, par = F.get_fd_coefficients(8), F.sim_params(c.dt, c.nt, c.dx, c.dz, 8)
src, rec = F.Source(60, 30, F.ricker_wavelet(c.f0, c.dt, c.nt)), F.setup_receivers(c.rec_x, c.rec_z, med)
submit = lambda srv, p=par, r=rec: srv.submit(med, H, a, src, r, p)
def wait(srv, t):
    try:
        srv.wait(t, timeout=60)
        return ""
    except F._lib.FomoError as e:
        return str(e)
med.upload()
"""


def test_failed_server_leaves_no_device_memory(host_run):
    host_run(SERVED + """
before = get("live_bytes")
for failing in ("fail_encode", "fail_alloc_min"):
    with F.ShotServer() as srv:
        t0 = submit(srv)
        assert wait(srv, t0) == ""
        put("fail_alloc_max", 1 << 40); put(failing, 1)
        assert "failed" in wait(srv, submit(srv))
        put("fail_encode", 0); put("fail_alloc_min", -1)
        try:
            submit(srv)
            raise AssertionError("a failed server took a shot")
        except F._lib.FomoError as e:
            assert "server failed" in str(e)
    assert get("live_bytes") == before, failing
with F.ShotServer() as srv:
    assert wait(srv, submit(srv)) == ""
""")


def test_library_shutdown_while_a_server_closes(host_run):
    host_run(SERVED + """
srv = F.ShotServer()
assert wait(srv, submit(srv)) == ""
put("hold_free", 1)
t = threading.Thread(target=srv.close)
t.start()
while not get("in_free"):                                 # the server has left the table of servers
    time.sleep(0.001)
down = threading.Thread(target=lambda: F._lib.call("fomo_b200_shutdown"))
down.start()
time.sleep(0.2)
put("hold_free", 0)
t.join(); down.join()
assert get("bad_pool_calls") == 0 and get("pools") == 0
F._lib._inited_device = None
F._lib.ensure_init(0)                                     # and the library starts again
W = F.Wavefield(60, 40, b)
med = F.init_medium(c.vp, c.vs, c.rho, c.dx, c.dz, c.nbc, 8, b)
med.upload()
with F.ShotServer() as srv:
    assert wait(srv, submit(srv)) == ""
""")


def test_servers_keep_their_share_of_the_pool(host_run):
    """What an idle server mapped is neither in another's budget nor taken by the library."""
    host_run(SERVED + """
import re
def budget(srv):
    long = F.sim_params(c.dt, 1 << 26, c.dx, c.dz, 8)     # a gather of 1.3 GB
    try:
        submit(srv, long)
        raise AssertionError("took a shot larger than the device")
    except F._lib.FomoError as e:
        return int(re.search(r"HBM budget of (\\d+)", str(e)).group(1))
cap = get("reserved") + (200 << 20)
put("capacity", cap)
A = F.ShotServer(hbm_budget_bytes=100 << 20)
put("hold", 1)
ts = [submit(A) for _ in range(40)]
put("hold", 0)
assert all(wait(A, t) == "" for t in ts)
share = A.stats()["peak_bytes"]
free = (200 << 20) - share
assert share > 10 << 20
with F.ShotServer() as B:                                 # free memory only
    assert abs(budget(B) - 0.9 * free) < 1 << 20, (budget(B), share)
try:                                                      # the library may not have it either
    F.Wavefield(2048, (free + share // 2) // (10 * 4 * 2048), b)
    raise AssertionError("the library took a live server's memory")
except F._lib.FomoError as e:
    assert "FOMO_ENOMEM" in str(e)
W = F.Wavefield(2048, int(free * 0.95) // (10 * 4 * 2048), b)
put("hold", 1)
ts = [submit(A) for _ in range(40)]
put("hold", 0)
assert all(wait(A, t) == "" for t in ts)                  # its burst still fits
W.release()
A.close()
with F.ShotServer() as B:                                 # what a closed server mapped counts as free
    assert abs(budget(B) - 0.9 * (cap - get("reserved") + share)) < 1 << 20
""")


def test_memory_of_a_closed_server_is_bounded_beside_a_live_one(host_run):
    host_run(SERVED + """
A = F.ShotServer()
assert wait(A, submit(A)) == ""
share = A.stats()["peak_bytes"]
base = get("reserved")
put("scale", 1000)                                        # 0.9 GB a shot
with F.ShotServer() as B:
    put("hold", 1)
    ts = [submit(B) for _ in range(8)]
    put("hold", 0)
    assert all(wait(B, t) == "" for t in ts)
    assert get("reserved") - base > 4 << 30
put("scale", 1)
assert get("reserved") - base <= share + (2 << 30)
assert wait(A, submit(A)) == ""
A.close()
""")


def test_resident_grid_is_no_timed_choice_in_the_cache_file(host_run, tmp_path):
    """A grid that ran the resident kernel was not timed: where it does not fit, both other kernels are."""
    path = tmp_path / "tune.txt"
    host_run("""
for _ in range(2):
    s = OpenShot(case(), b)
    s.advance(600)
    s.finish()
""", FOMO_B200_TUNE_CACHE=str(path))
    assert path.read_text().split() == ["step", "182", "122", "4", "12", "1", "1", "0", "resident"]
    host_run("""
put("sm_count", 2)                                        # a device the grid's three strips do not fit
s = OpenShot(case(), b)
s.advance(600)
assert get("launches:resident_kernel") == 0
assert get("launches:" + MARCH) >= 24 and get("launches:" + SPLIT) >= 24
assert steps() == 600
""", FOMO_B200_TUNE_CACHE=str(path))
    lines = path.read_text().strip().split("\n")
    assert len(lines) == 2 and lines[1].split()[:7] == lines[0].split()[:7] and lines[1].split()[7] in ("0", "1")
    chosen = 600 if lines[1].split()[7] == "1" else 0
    host_run(f"""
put("sm_count", 2)                                        # the timed choice is read
s = OpenShot(case(), b)
s.advance(600)
assert get("launches:" + MARCH) == {chosen} and get("launches:" + SPLIT) == 600 - {chosen}
""", FOMO_B200_TUNE_CACHE=str(path))


def test_steps_per_launch_in_the_cache_file(host_run, tmp_path):
    """A K in the file is obeyed; the default is noted and not read as a choice."""
    path = tmp_path / "tune.txt"
    script = SERVED + """
with F.ShotServer() as srv:
    assert wait(srv, submit(srv, F.sim_params(c.dt, 64, c.dx, c.dz, 8))) == ""
print(get("launches:19batch_stress_kernel"))              # those of one captured graph
"""
    assert host_run(script, FOMO_B200_TUNE_CACHE=str(path)).split() == ["8"]
    assert path.read_text() == "182 122 4 0 8 default\n"
    path.write_text("182 122 4 0 32 default\n")
    assert host_run(script, FOMO_B200_TUNE_CACHE=str(path)).split() == ["8"]
    path.write_text("182 122 4 0 32\n")
    assert host_run(script, FOMO_B200_TUNE_CACHE=str(path)).split() == ["32"]
    assert path.read_text() == "182 122 4 0 32\n"
