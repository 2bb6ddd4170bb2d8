"""One shot over several time-step kernels: whichever kernels its calls run
(the process-wide selection can change between two of them, and a profiled
call runs the split launches), the gather and the wavefield are those of the
shot run by one kernel, bit for bit."""
import ctypes

import numpy as np
import pytest

import fomo_julia_b200 as F
from fomo_julia_b200 import elastic2d
from fomo_julia_b200._lib import FomoKernelTime, FomoRunStats, call
from cases import layered

pytestmark = pytest.mark.gpu
FIELDS = ("vx", "vz", "txx", "tzz", "txz")


@pytest.fixture
def step_kernel():
    """Selects the time-step kernels for one test and restores "auto"."""
    yield F.set_step_kernel
    F.set_step_kernel("auto")


class OpenShot:
    """A shot of a case, advanced call by call."""

    def __init__(self, c, b200):
        self.med = F.init_medium(c.vp, c.vs, c.rho, c.dx, c.dz, c.nbc, c.fd_order, b200, free_surface=c.free_surface)
        H = F.init_habc(self.med.nx, self.med.nz, c.nbc, c.dt, c.dx, c.dz, c.v_ref, b200)
        src = F.Source(F.coord_to_index(c.src_x, c.dx, self.med.pad), F.coord_to_index(c.src_z, c.dz, self.med.pad),
                       F.ricker_wavelet(c.f0, c.dt, c.nt))
        rec = F.setup_receivers(c.rec_x, c.rec_z, self.med, type=c.rec_type)
        self.W = F.Wavefield(self.med.nx, self.med.nz, b200)
        keep = []
        hs = elastic2d._ctypes_habc(H, keep)
        ss = elastic2d._ctypes_shot(F.get_fd_coefficients(c.fd_order), F.sim_params(c.dt, c.nt, c.dx, c.dz, c.fd_order),
                                    src, rec, keep)
        self.gather = np.zeros((c.nt, ss.n_rec), dtype=np.float32, order="F")
        self.handle, self.k = ctypes.c_uint64(0), ctypes.c_int32(0)
        call("fomo_b200_shot_begin", self.med.upload(), self.W.handle, ctypes.byref(hs), ctypes.byref(ss),
             ctypes.byref(self.handle))

    def advance(self, n):
        call("fomo_b200_shot_advance", self.handle.value, n, ctypes.byref(self.k))

    def profile(self, n):
        kt, nk = (FomoKernelTime * 5)(), ctypes.c_int32(0)
        call("fomo_b200_shot_profile", self.handle.value, n, kt, 5, ctypes.byref(nk))
        return {kt[q].name.decode(): kt[q].launches for q in range(nk.value)}

    def finish(self):
        """(gather, fields, kernel launches)"""
        st = FomoRunStats()
        fields = {f: self.W.field(f) for f in FIELDS}
        call("fomo_b200_shot_finish", self.handle.value, self.gather.ctypes.data, ctypes.byref(st))
        self.W.release()
        self.med.release()
        return self.gather, fields, st.kernel_launches


def whole_shot(c, b200, step_kernel, mode):
    step_kernel(mode)
    s = OpenShot(c, b200)
    s.advance(c.nt)
    return s.finish()


def assert_equal(a, b):
    assert np.array_equal(a[0], b[0]), f"gather rows {np.unique(np.nonzero(a[0] != b[0])[0])} differ"
    for f in FIELDS:
        assert np.array_equal(a[1][f], b[1][f]), f


# calls of one shot: (kernels selected or "profile", steps)
ROUTES = {
    "profile-auto-split-auto": [("profile", 20), ("auto", 20), ("split", 10), ("auto", 60)],
    "fused-auto-split-fused": [("fused", 7), ("auto", 33), ("split", 1), ("fused", 60)],
    "split-auto": [("split", 1), ("auto", 80)],
    "auto-profile-finish": [("auto", 40), ("profile", 24)],
}


@pytest.mark.parametrize("rec_type", ["vz", "p"])
@pytest.mark.parametrize("route", list(ROUTES.values()), ids=list(ROUTES))
def test_kernels_change_within_a_shot(route, rec_type, b200, step_kernel):
    c = layered(150, 90, seed=4, nbc=12, fd_order=8, nt=64, rec_type=rec_type)
    ref = whole_shot(c, b200, step_kernel, "split")
    assert (np.abs(ref[0]).max(axis=1) > 0).sum() >= 60  # rows that a lost one would differ from
    s = OpenShot(c, b200)
    for mode, n in route:
        if mode == "profile":
            step_kernel("auto")
            s.profile(n)
        else:
            step_kernel(mode)
            s.advance(n)
    assert s.k.value == c.nt or route[-1][0] == "profile"
    assert_equal(s.finish(), ref)


def test_saved_gather_after_a_change_of_kernels(b200, step_kernel, tmp_path):
    c = layered(150, 90, seed=4, nbc=12, fd_order=8, nt=64)
    ref = whole_shot(c, b200, step_kernel, "split")
    s = OpenShot(c, b200)
    s.advance(30)
    step_kernel("auto")
    s.advance(34)
    path = tmp_path / "g.bin"
    call("fomo_b200_shot_save_gather", s.handle.value, str(path).encode())
    s.finish()
    assert np.array_equal(F.load_gather(str(path), *ref[0].shape), ref[0])


def test_kernels_timed_on_live_steps(b200, step_kernel, tmp_path, monkeypatch):
    """A grid too large for the resident kernel: its first shot times the fused step and the split launches on 24
    steps each, records the faster and runs the rest on it."""
    path = tmp_path / "tune.txt"
    monkeypatch.setenv("FOMO_B200_TUNE_CACHE", str(path))
    c = layered(1463, 883, seed=6, nbc=10, fd_order=8, nt=100, n_rec=9)  # 1491 x 911 padded
    first = whole_shot(c, b200, step_kernel, "auto")
    line = path.read_text().split()
    assert line[:7] == ["step", "1491", "911", "4", "10", "1", "1"] and line[7:] in (["0"], ["1"])
    rest = 1 if line[7] == "1" else 4  # launches per step
    assert first[2] == 24 + 4 * 24 + rest * 52 + 1  # and the last row's receivers
    again = whole_shot(c, b200, step_kernel, "auto")
    assert again[2] == rest * 100 + 1 and path.read_text().split() == line
    ref = whole_shot(c, b200, step_kernel, "split")
    assert ref[2] == 401 and np.abs(ref[0]).max() > 0
    assert_equal(first, ref)
    assert_equal(again, ref)
