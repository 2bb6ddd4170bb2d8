"""The resident kernel (many time steps per launch, fields in shared memory)
against the oracle, bit for bit, at the sizes where its layout changes: one,
two and several column strips, one and several rows of blocks, every order,
HABC bands from 1 layer to the widest it takes, sources on block borders,
more receivers than a block lists, and runs longer than one launch."""
import dataclasses
import threading

import numpy as np
import pytest

import fomo_julia_b200 as F
from cases import layered, oracle_inputs

pytestmark = pytest.mark.gpu
FIELDS = ("vx", "vz", "txx", "tzz", "txz")
STEPS_PER_LAUNCH = 256


def _run(c, b200, on_step=None, step_chunk=1, wavelet=None):
    med = F.init_medium(c.vp, c.vs, c.rho, c.dx, c.dz, c.nbc, c.fd_order, b200, free_surface=c.free_surface)
    H = F.init_habc(med.nx, med.nz, c.nbc, c.dt, c.dx, c.dz, c.v_ref, b200)
    wav = F.ricker_wavelet(c.f0, c.dt, c.nt) if wavelet is None else wavelet
    rec = F.setup_receivers(c.rec_x, c.rec_z, med, type=c.rec_type)
    src = F.Source(F.coord_to_index(c.src_x, med.dx, med.pad), F.coord_to_index(c.src_z, med.dz, med.pad), wav)
    W = F.Wavefield(med.nx, med.nz, b200)
    r = F.run_shot(b200, W, med, H, F.get_fd_coefficients(c.fd_order), src, rec,
                   F.sim_params(c.dt, c.nt, c.dx, c.dz, c.fd_order), on_step=on_step, step_chunk=step_chunk)
    fields = {f: W.field(f) for f in FIELDS}
    W.release()
    med.release()
    return r, fields


def _check(c, b200, oracle_lib, wavelet=None, **kw):
    r, f = _run(c, b200, wavelet=wavelet, **kw)
    med, h, a, wav, si, sj, ri, rj = oracle_inputs(c, oracle_lib)
    wav = wav if wavelet is None else np.asarray(wavelet, dtype=wav.dtype)
    g, fin = oracle_lib.run_shot(med, h, a, c.dt, c.nt, si, sj, wav, ri, rj, c.rec_type, "simd8", final_fields=True)
    assert np.abs(g).max() > 0 or np.abs(fin).max() > 0
    assert np.array_equal(r.gather, g)
    for q, name in enumerate(FIELDS):
        assert np.array_equal(f[name], fin[:, :, q]), f"{name}: {np.count_nonzero(f[name] != fin[:, :, q])} cells differ"
    return r


# (nx_in, nz_in, order, nbc, free surface): padded sizes nx_in + 2 (nbc + order / 2)
SHAPES = [
    (20, 14, 8, 5, True),       # one strip, one or two rows of blocks
    (24, 20, 12, 2, False),     # bands shorter than the stencil
    (30, 22, 2, 1, False),      # one HABC layer, half stencil of one cell (rows of 8)
    (50, 40, 10, 3, True),
    (46, 33, 8, 5, False),      # exactly one strip of 64 columns
    (47, 33, 8, 5, True),       # one column more
    (100, 30, 4, 12, True),     # two strips
    (131, 300, 6, 7, True),     # three strips, many rows of blocks
    (201, 160, 8, 59, True),    # widest bands with strips of 64 (60 columns needed)
    (141, 90, 8, 33, False),
    (640, 41, 8, 20, True),     # wide and shallow
    (37, 700, 4, 9, False),     # narrow and deep
    (900, 500, 12, 30, True),   # tall regions: two rows per thread, medium in global memory
    (700, 420, 2, 44, False),
]


@pytest.mark.parametrize("nx,nz,order,nbc,fs", SHAPES, ids=lambda v: str(v))
def test_resident_shapes(nx, nz, order, nbc, fs, b200, oracle_lib):
    nt = 70 if nx * nz < 100000 else 40
    c = layered(nx, nz, seed=nx + order, nbc=nbc, fd_order=order, free_surface=fs, nt=nt, n_rec=11,
                rec_type=("vz", "vx", "p")[nx % 3])
    r = _check(c, b200, oracle_lib)
    assert r.stats["kernel_launches"] <= 2


def test_resident_anisotropic_grid(b200, oracle_lib):
    c = layered(180, 120, seed=3, nbc=10, fd_order=8, nt=80)
    c = dataclasses.replace(c, dz=13.0)
    assert _check(c, b200, oracle_lib).stats["kernel_launches"] <= 2


@pytest.mark.parametrize("rec_type", ["p", "vx"])
@pytest.mark.parametrize("di,dj", [(0, 0), (-20, 4), (-6, -6), (3, 60)])
def test_resident_source_and_receivers_anywhere(di, dj, rec_type, b200, oracle_lib):
    """Sources at the first cells of blocks, in the bands and on the free surface, a receiver on the source."""
    c = layered(170, 100, seed=5, nbc=16, fd_order=8, nt=60, n_rec=9)
    c.src_x = float(c.dx) * (60 - 20 + di)  # padded columns 60 + di and so on (pad 20)
    c.src_z = float(c.dz) * (15 - 20 + 30 + dj)
    c.rec_x = np.append(c.rec_x, np.float32(c.src_x))
    c.rec_z = np.append(c.rec_z, np.float32(c.src_z))
    c.rec_type = rec_type
    _check(c, b200, oracle_lib)


def test_resident_many_receivers_and_launches(b200, oracle_lib):
    """More receivers in one block than it lists, a wavelet shorter than the run, more than one launch."""
    c = layered(60, 40, seed=9, nbc=6, fd_order=8, nt=2 * STEPS_PER_LAUNCH + 17, n_rec=900)
    c.rec_x = np.full(900, 200.0, dtype=np.float32)
    wav = F.ricker_wavelet(c.f0, c.dt, c.nt)[:300]
    r = _check(c, b200, oracle_lib, wavelet=wav)
    assert r.stats["kernel_launches"] == 3
    seen = []
    chunked, _ = _run(c, b200, on_step=lambda W, info: seen.append(W.snapshot("p", 2).shape), step_chunk=100, wavelet=wav)
    assert len(seen) == 6 and np.array_equal(chunked.gather, r.gather)


def test_resident_beside_a_busy_server(b200, oracle_lib):
    """Single shots on the resident kernel while a server's launches keep the GPU busy."""
    big = layered(900, 500, seed=2, nbc=20, fd_order=8, nt=400, n_rec=5)
    med = F.init_medium(big.vp, big.vs, big.rho, big.dx, big.dz, big.nbc, big.fd_order, b200)
    H = F.init_habc(med.nx, med.nz, big.nbc, big.dt, big.dx, big.dz, big.v_ref, b200)
    wav = F.ricker_wavelet(big.f0, big.dt, big.nt)
    rec = F.setup_receivers(big.rec_x, big.rec_z, med)
    src = F.Source(med.nx // 2, med.pad + 3, wav)
    params = F.sim_params(big.dt, big.nt, big.dx, big.dz, big.fd_order)
    c = layered(150, 90, seed=4, nbc=12, fd_order=8, nt=300)
    ref, _ = _run(c, b200)
    out = []
    with F.ShotServer() as srv:
        ts = [srv.submit(med, H, F.get_fd_coefficients(8), src, rec, params) for _ in range(40)]
        t = threading.Thread(target=lambda: out.extend(_run(c, b200)[0] for _ in range(5)))
        t.start()
        res = srv.wait_all(ts, timeout=120.0)
        t.join()
    assert len(out) == 5 and all(np.array_equal(r.gather, ref.gather) for r in out)
    assert all(np.array_equal(r.gather, res[0].gather) for r in res)
    med.release()


def test_resident_wait_is_bounded(b200, oracle_lib):
    """A wait for a message that nobody sends ends with FOMO_ETIMEOUT, whatever the limit, and a shot runs after it."""
    import ctypes
    from fomo_julia_b200._lib import call, load
    st = ctypes.c_int32(0)
    for polls in (1, 1000, 4097):
        call("fomo_b200_selftest_wait", polls, ctypes.byref(st))
        assert st.value == -4
        assert b"did not hear from its neighbours" in load().fomo_b200_last_error()
    _check(layered(50, 40, seed=7, nbc=5, fd_order=8, nt=60), b200, oracle_lib)
