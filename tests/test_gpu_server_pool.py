"""The servers' shared memory pool: batches made again and again, and servers
side by side in threads, give the gathers of the first, and what a closed
server held is available to the next one's budget."""
import threading

import numpy as np
import pytest

import fomo_julia_b200 as F
from cases import layered

pytestmark = pytest.mark.gpu


def _survey(b200, n, seed):
    c = layered(150, 80, seed=seed, nbc=10, fd_order=8, nt=60, n_rec=9)
    med = F.init_medium(c.vp, c.vs, c.rho, c.dx, c.dz, c.nbc, c.fd_order, b200)
    H = F.init_habc(med.nx, med.nz, c.nbc, c.dt, c.dx, c.dz, c.v_ref, b200)
    rec = F.setup_receivers(c.rec_x, c.rec_z, med)
    cfg = F.multi_shot_config([300.0 + 40 * k for k in range(n)], [20.0] * n, F.ricker_wavelet(c.f0, c.dt, c.nt))
    return med, lambda: [r.gather for r in F.run_batch(b200, med, H, F.get_fd_coefficients(8), rec, cfg,
                                                       F.sim_params(c.dt, c.nt, c.dx, c.dz, 8))]


def test_batches_reuse_the_pool(b200):
    med, run = _survey(b200, 14, 3)
    first = run()
    assert np.abs(first[0]).max() > 0
    for _ in range(4):
        assert all(np.array_equal(a, b) for a, b in zip(run(), first))
    med.release()


def test_servers_side_by_side(b200):
    surveys = [_survey(b200, n, seed) for n, seed in ((13, 4), (5, 5), (26, 6))]
    ref = [run() for _, run in surveys]
    out = [[] for _ in surveys]

    def work(k):
        out[k] += [surveys[k][1]() for _ in range(4)]

    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(surveys))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, runs in enumerate(out):
        assert len(runs) == 4
        for r in runs:
            assert all(np.array_equal(a, b) for a, b in zip(r, ref[k]))
        surveys[k][0].release()


@pytest.mark.parametrize("ds", [1, 3])
def test_frames_through_pinned_memory(ds, b200):
    """Frames below and above the pinned buffer's 4 MB are the fields' values."""
    for nx, nz in ((61, 47), (1300, 1100)):
        W = F.Wavefield(nx, nz, b200)
        v = np.asfortranarray(np.random.default_rng(nx).standard_normal((nx, nz)).astype(np.float32))
        W.set_field("vx", v)
        assert np.array_equal(W.snapshot("vx", ds), v[::ds, ::ds])
        W.release()
