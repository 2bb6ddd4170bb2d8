"""Performance cases: what users of this package have it do, at the sizes they do it.

Every case is one call (or one stream of requests) of the public API on media
and survey layouts made here from a seed:

* ``shot``   one ``run_shot``: wavefield reset, nt time steps, gather on the host;
* ``movie``  one ``run_shot`` with an ``on_step`` snapshot recorder every `skip` steps;
* ``batch``  one ``run_shots(batched=True)``: many shots on one medium;
* ``serve``  a burst of requests over several media to a running ``ShotServer``.

The media are layered models with smooth perturbations (and a water layer
where the case says so), the shape of the workloads in
``fomo_julia_b200.synthetic``.  ``exact`` evaluates the same scheme in Float64
with plain torch.
"""
import math

import numpy as np
import torch

import fomo_julia_b200 as F

f32 = np.float32


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _shot(name, nx, nz, order, nbc, nt, n_rec, rec="vz", fs=True, water=0, aniso=False, kind="shot", **more):
    return dict(name=name, kind=kind, nx=nx, nz=nz, order=order, nbc=nbc, nt=nt, n_rec=n_rec, rec=rec, fs=fs,
                water=water, aniso=aniso, **more)


def listed():
    return [
        # a first try or a regression check on a small model: latency per step is all there is
        _shot("shot_160x80_o8", 160, 80, 8, 20, 400, 40),
        # the small homogeneous-size survey of the benchmark (400 x 200, nt 1500, 199 receivers), vx
        _shot("shot_400x200_o8", 400, 200, 8, 50, 1500, 199, rec="vx"),
        # the uneven batch's smallest grid, odd, order 4, pressure under water
        _shot("shot_601x301_o4_p", 601, 301, 4, 50, 1500, 150, rec="p", water=15),
        # no free surface (a buried or fully absorbing model), order 6, dx != dz
        _shot("shot_843x397_o6_nofs", 843, 397, 6, 30, 1000, 211, fs=False, aniso=True),
        # the uneven batch's second grid at its highest order
        _shot("shot_1200x500_o12", 1200, 500, 12, 50, 1000, 400),
        # one shot of the 2000 x 800 survey
        _shot("shot_2000x800_o8", 2000, 800, 8, 50, 1500, 400, water=12),
        # the uneven batch's largest grid
        _shot("shot_3200x1400_o8", 3200, 1400, 8, 50, 800, 800, water=15),
        # the large layered shot of the benchmark (fewer steps)
        _shot("shot_4444x3819_o8", 4444, 3819, 8, 50, 1000, 1000, water=15),
        # wavefield movie: a frame of p every 10 steps, as the video recorder takes them
        _shot("movie_1000x400_o8", 1000, 400, 8, 50, 600, 200, kind="movie", skip=10, downsample=2),
        # a small survey in one batch: 24 shots on the 400 x 200 model
        _shot("batch_400x200_24shots", 400, 200, 8, 50, 800, 199, kind="batch", shots=24),
        # a part of the 64-shot survey on the 2000 x 800 medium
        _shot("batch_2000x800_16shots", 2000, 800, 8, 50, 400, 400, kind="batch", shots=16, water=12),
        # a burst of uneven requests (orders 4/8/12, the uneven batch's media) to a running server
        _shot("serve_mixed_20", 2400, 1000, 8, 50, 500, 400, kind="serve", shots=20, media=3),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["shot"] * 6 + ["movie", "batch", "batch", "serve"])
    top = {"shot": 4400, "movie": 2400, "batch": 2200, "serve": 2200}[kind]
    nx = log_int(150, top)
    nz = max(64, min(3800, int(nx * rng.uniform(0.35, 0.95))))
    nbc = rng.randint(10, 50)
    order = rng.choice([2, 4, 4, 6, 8, 8, 8, 8, 10, 12])
    shots = {"shot": 1, "movie": 1, "batch": rng.randint(2, 24), "serve": rng.randint(4, 24)}[kind]
    cells = (nx + 2 * nbc + order) * (nz + 2 * nbc + order)
    nt = max(120, min(rng.randint(300, 2000), int(6.0e9 / (cells * shots))))
    c = _shot("", nx, nz, order, nbc, nt, log_int(10, 1000), rec=rng.choice(["vz", "vz", "vx", "p"]),
              fs=rng.random() < 0.8, water=rng.choice([0, 0, min(15, nz // 20)]), aniso=rng.random() < 0.25, kind=kind)
    if kind == "movie":
        c.update(skip=rng.randint(5, 25), downsample=rng.randint(1, 4))
    if kind in ("batch", "serve"):
        c.update(shots=shots)
    if kind == "serve":
        c.update(media=rng.randint(2, 4))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _model(nx, nz, water, seed):
    """vp, vs, rho as (nx, nz) Float32 arrays, x fastest: layers of rising
    velocity times a smooth random perturbation, under `water` rows of water."""
    g = torch.Generator().manual_seed(seed)
    coarse = torch.randn(1, 1, nz // 20 + 3, nx // 20 + 3, generator=g).to(_device())
    p = torch.nn.functional.interpolate(coarse, size=(nz, nx), mode="bicubic", align_corners=True)[0, 0]
    p = p / p.abs().max()
    n_layers = max(3, min(40, nz // 12))
    layer = torch.div(torch.arange(nz, device=p.device) * n_layers, nz, rounding_mode="floor")
    vp = (1800.0 + 2700.0 * layer.float() / (n_layers - 1))[:, None] * (1.0 + 0.05 * p)
    vs = vp / 1.73
    if water:
        vp[:water] = 1500.0
        vs[:water] = 0.0
    rho = 310.0 * vp ** 0.25
    return tuple(t.to(torch.float32).cpu().numpy().T for t in (vp, vs, rho))


def _coefficients(order):
    """Staggered-grid Taylor coefficients, rounded to Float32."""
    M = order // 2
    k = 2 * np.arange(M)[:, None] + 1.0
    odd = 2 * np.arange(M)[None, :] + 1.0
    return np.linalg.solve(odd ** k, np.eye(M)[0]).astype(f32)


def _ricker(f0, dt, nt):
    t = np.arange(nt) * float(dt) - 1.0 / f0
    x = (np.pi * f0 * t) ** 2
    return ((1.0 - 2.0 * x) * np.exp(-x)).astype(f32)


def _length(c, s):
    """Steps and receivers of shot s: a server's requests run 0.6 to 1 times
    the case's steps and 0.5 to 1 times its receivers."""
    if c["kind"] != "serve":
        return c["nt"], c["n_rec"]
    return int(c["nt"] * (0.6 + 0.4 * (7 * s % 10) / 9)), max(1, int(c["n_rec"] * (0.5 + 0.5 * (3 * s % 10) / 9)))


def _survey(c, seed):
    """Everything a case's calls take, as plain values: media and requests."""
    rng = np.random.default_rng(seed)
    media, jobs = [], []
    for m in range(c.get("media", 1)):
        # a server's further media are smaller ones of other orders
        nx, nz = max(150, c["nx"] >> m), max(64, c["nz"] >> m)
        order = c["order"] if m == 0 else (4, 12, 8)[(m - 1) % 3]
        dx = 10.0
        dz = 12.5 if c["aniso"] else 10.0
        vp, vs, rho = _model(nx, nz, c["water"] >> m, 1000 * seed + m)
        dt = f32(0.45 * dx / float(vp.max()))
        media.append(dict(vp=vp, vs=vs, rho=rho, nx=nx, nz=nz, order=order, nbc=c["nbc"], fs=c["fs"], dx=dx, dz=dz,
                          dt=dt, v_ref=f32(vp.mean(dtype=np.float64)), a=_coefficients(order)))
    for s in range(c.get("shots", 1)):
        m = s % len(media)
        d = media[m]
        uneven = c["kind"] == "serve"
        nt, n_rec = _length(c, s)
        span = (d["nx"] - 1) * d["dx"]
        f0 = 1500.0 / (8.0 * d["dx"]) * (rng.uniform(0.7, 1.0) if uneven or s == 0 else 1.0)
        if s and not uneven:
            f0 = jobs[0]["f0"]  # a survey's shots share their wavelet and receivers
        # a source a few cells beside one of the receivers, which record it from the first steps on
        rec_x = np.linspace(0.0, span, n_rec).astype(f32)
        src_x = f32(min(span, rec_x[rng.integers(0, n_rec)] + d["dx"] * rng.integers(0, 8)))
        rec_z = 2 + (c["water"] >> m)
        jobs.append(dict(medium=m, nt=nt, f0=f0, wavelet=_ricker(f0, d["dt"], nt),
                         src_x=src_x, src_z=f32(d["dz"] * (3 if d["fs"] else 12)), rec_x=rec_x,
                         rec_z=np.full(n_rec, rec_z * d["dz"], dtype=f32), rec=c["rec"]))
    return media, jobs


class _State:
    """What a user's program keeps between calls; released with the object."""

    def __init__(self, case):
        self.case, self.backend = case, F.backend("b200")
        self.media, self.habc, self.jobs = [], [], []
        self.wavefield = self.server = None

    def __del__(self):
        if self.server is not None:
            self.server.close()
        if self.wavefield is not None:
            self.wavefield.release()
        for m in self.media:
            m.release()


def prepare(case, seed):
    media, jobs = _survey(case, seed)
    s = _State(case)
    s.data = media
    for d in media:
        m = F.init_medium_device(d["vp"], d["vs"], d["rho"], d["dx"], d["dz"], d["nbc"], d["order"], s.backend,
                                 free_surface=d["fs"])
        s.media.append(m)
        s.habc.append(F.init_habc(m.nx, m.nz, d["nbc"], d["dt"], d["dx"], d["dz"], d["v_ref"], s.backend))
    for j in jobs:
        d, m = media[j["medium"]], s.media[j["medium"]]
        s.jobs.append(dict(
            j, params=F.sim_params(d["dt"], j["nt"], d["dx"], d["dz"], d["order"]),
            source=F.Source(F.coord_to_index(j["src_x"], m.dx, m.pad), F.coord_to_index(j["src_z"], m.dz, m.pad),
                            j["wavelet"]),
            receivers=F.setup_receivers(j["rec_x"], j["rec_z"], m, type=j["rec"])))
    if case["kind"] in ("shot", "movie"):
        s.wavefield = F.Wavefield(s.media[0].nx, s.media[0].nz, s.backend)
    if case["kind"] == "batch":
        s.config = F.multi_shot_config([j["src_x"] for j in jobs], [j["src_z"] for j in jobs], jobs[0]["wavelet"])
    if case["kind"] == "serve":
        s.server = F.ShotServer()
    return s


# ---------------------------------------------------------------------------
# The calls
# ---------------------------------------------------------------------------
def run(s):
    kind, j = s.case["kind"], s.jobs[0]
    if kind == "shot":
        r = F.run_shot(s.backend, s.wavefield, s.media[0], s.habc[0], s.data[0]["a"], j["source"], j["receivers"],
                       j["params"])
        return {"gather": r.gather}
    if kind == "movie":
        film = F.SnapshotRecorder(F.VideoConfig(fields=("p",), skip=s.case["skip"], downsample=s.case["downsample"]))
        r = F.run_shot(s.backend, s.wavefield, s.media[0], s.habc[0], s.data[0]["a"], j["source"], j["receivers"],
                       j["params"], on_step=film, step_chunk=s.case["skip"])
        return {"gather": r.gather, "frames": film.stack("p")}
    if kind == "batch":
        rs = F.run_shots(s.backend, None, s.media[0], s.habc[0], s.data[0]["a"], j["receivers"], s.config,
                         j["params"], batched=True)
        return {"gathers": [r.gather for r in rs]}
    tickets = [s.server.submit(s.media[q["medium"]], s.habc[q["medium"]], s.data[q["medium"]]["a"], q["source"],
                               q["receivers"], q["params"], shot_id=k + 1) for k, q in enumerate(s.jobs)]
    return {"gathers": [r.gather for r in s.server.wait_all(tickets)]}


def _grids(case):
    """(padded nx, padded nz, half stencil width) of each medium, and (medium, steps, receivers) of each shot."""
    grids = []
    for m in range(case.get("media", 1)):
        order = case["order"] if m == 0 else (4, 12, 8)[(m - 1) % 3]
        pad = case["nbc"] + order // 2
        grids.append((max(150, case["nx"] >> m) + 2 * pad, max(64, case["nz"] >> m) + 2 * pad, order // 2))
    return grids, [(s % len(grids), *_length(case, s)) for s in range(case.get("shots", 1))]


def work(case):
    """Per time step: the five fields read and written (40 B a cell, each
    shot) and the five medium arrays read (20 B a cell, once for the shots
    of a medium that run side by side); the scheme's additions and
    multiplications (3 for each of the 8 derivatives' M terms, 25 for the
    updates).  The gathers once, and a movie's frames."""
    grids, shots = _grids(case)
    b = fl = 0.0
    for m, (nx, nz, M) in enumerate(grids):
        cells = float(nx) * nz
        mine = [(nt, n_rec) for g, nt, n_rec in shots if g == m]
        b += sum(40.0 * cells * nt + 4.0 * nt * n_rec for nt, n_rec in mine)
        b += 20.0 * cells * max([nt for nt, _ in mine], default=0)
        fl += sum((24.0 * M + 25.0) * cells * nt for nt, _ in mine)
    if case["kind"] == "movie":
        nx, nz, _ = grids[0]
        d = case["downsample"]
        b += (case["nt"] // case["skip"]) * 4.0 * math.ceil(nx / d) * math.ceil(nz / d)
    return {"bytes": b, "flops": fl}


# ---------------------------------------------------------------------------
# The same scheme in Float64
# ---------------------------------------------------------------------------
class _Exact:
    """Shots on one medium in Float64, fields as (shot, z, x) tensors."""

    def __init__(self, d, jobs):
        dev = _device()
        t = lambda x: torch.from_numpy(np.ascontiguousarray(x, dtype=np.float64)).to(dev)  # noqa: E731
        self.M, self.b, self.fs = d["order"] // 2, d["nbc"], d["fs"]
        self.pad = self.M + self.b
        p, M, b = self.pad, self.M, self.b
        vp, vs, rho = (torch.nn.functional.pad(t(d[k].T)[None, None], (p, p, p, p), mode="replicate")[0, 0]
                       for k in ("vp", "vs", "rho"))
        mu = rho * vs * vs
        self.lam, self.mu, self.rx = rho * vp * vp - 2 * mu, mu, rho
        self.rz, self.mxz = torch.zeros_like(rho), torch.zeros_like(mu)
        self.rz[:-1, :-1] = 0.25 * (rho[:-1, :-1] + rho[:-1, 1:] + rho[1:, :-1] + rho[1:, 1:])
        self.rz[:, -1] = self.rz[:, -2]
        self.rz[-1] = self.rz[-2]
        self.mxz[:-1] = 2.0 / (1.0 / mu[:-1] + 1.0 / mu[1:])
        self.mxz[-1] = self.mxz[-2]
        self.nz, self.nx = rho.shape
        nx, nz = self.nx, self.nz
        dt = float(d["dt"])
        self.dtx, self.dtz = dt / d["dx"], dt / d["dz"]
        self.a = [float(x) for x in d["a"]]
        # HABC: one-way extrapolation coefficients and blending weights by distance to the edge
        rx, rz = float(d["v_ref"]) * self.dtx, float(d["v_ref"]) * self.dtz
        q = lambda r, s: (0.45 * (1 + r) - s) / ((1 + r) * 0.55)  # noqa: E731
        self.qx, self.qz, self.qtx, self.qtz, self.qxt = q(rx, rx), q(rz, rz), q(rx, 1.0), q(rz, 1.0), 0.45 / -0.55
        i, j = torch.arange(nx, device=dev), torch.arange(nz, device=dev)
        dist = torch.minimum(torch.minimum(i, nx - 1 - i)[None], torch.minimum(j, nz - 1 - j)[:, None]).double()
        self.w = {k: ((dist - off) / b).clamp(0, 1) for k, off in (("vx", 0.0), ("vz", 0.5), ("t", 0.75))}
        # bottom band: f[j] = A[j] + B[j] f[j-1], solved as a product with the recurrence's matrix
        self.P = {}
        for k, w in self.w.items():
            B = -(1 - w[nz - b - 1:nz - 1]) * self.qz
            corner = (i <= b) | (i >= nx - b - 1)
            B[:, corner] *= 0.5
            cols = torch.cat([torch.nonzero(corner)[:, 0], torch.tensor([b + 1], device=dev)])
            Bc = B[:, cols]
            P = torch.zeros(cols.numel(), b, b + 1, dtype=torch.float64, device=dev)
            for r in range(b):
                P[:, r, r + 1] = 1.0
                P[:, r, :r + 1] = (P[:, r - 1, :r + 1] if r else 1.0) * Bc[r][:, None]
            self.P[k] = (cols[:-1], P[:-1], P[-1])
        S = len(jobs)
        self.f = {k: torch.zeros(S, nz, nx, dtype=torch.float64, device=dev) for k in ("vx", "vz", "xx", "zz", "xz")}
        idx = lambda x, h: np.rint(np.asarray(x, dtype=f32) / f32(h)).astype(np.int64) + p  # noqa: E731
        self.S = torch.arange(S, device=dev)
        self.si = torch.tensor([int(idx(q["src_x"], d["dx"])) for q in jobs], device=dev)
        self.sj = torch.tensor([int(idx(q["src_z"], d["dz"])) for q in jobs], device=dev)
        self.ri = torch.from_numpy(np.stack([idx(q["rec_x"], d["dx"]) for q in jobs])).to(dev)
        self.rj = torch.from_numpy(np.stack([idx(q["rec_z"], d["dz"]) for q in jobs])).to(dev)
        self.kind = jobs[0]["rec"]
        self.wav = torch.stack([t(q["wavelet"]) for q in jobs], 1)

    def diff(self, f, axis, s):
        """sum_l a_l (f[k+l-1+s] - f[k-l+s]) along an axis (1 z, 2 x), on the interior."""
        M, nx, nz = self.M, self.nx, self.nz
        cut = lambda o: (f[:, M + o:nz - M + o, M:nx - M] if axis == 1 else f[:, M:nz - M, M + o:nx - M + o])  # noqa: E731
        out = None
        for n, a in enumerate(self.a):
            out = (cut(n + s) - cut(s - n - 1)) * a if out is None else out.add_(cut(n + s) - cut(s - n - 1), alpha=a)
        return out

    def edge(self, f, o, w, dst, nb, q, qt):
        """The blended one-way value of an edge region; dst and nb index (z, x)."""
        d, n = (slice(None),) + dst, (slice(None),) + nb
        return w[dst] * f[d] + (1 - w[dst]) * (-q * f[n] - qt * o[d] - self.qxt * o[n])

    def habc(self, f, o, key):
        b, nx, nz = self.b, self.nx, self.nz
        w = self.w[key]
        r0, j0, js = nx - b - 1, nz - b - 1, (self.b if self.fs else 1)
        pre = f.clone()
        rows = slice(js, j0)
        # left: neighbours before the update; right: chunks of 8, a chunk's first column reads the updated one before it
        f[:, rows, 1:b + 1] = self.edge(pre, o, w, (rows, slice(1, b + 1)), (rows, slice(2, b + 2)), self.qx, self.qtx)
        f[:, rows, r0:nx - 1] = self.edge(pre, o, w, (rows, slice(r0, nx - 1)), (rows, slice(r0 - 1, nx - 2)), self.qx, self.qtx)
        if r0 + 8 < nx - 1:
            c, n = slice(r0 + 8, nx - 1, 8), slice(r0 + 7, nx - 2, 8)
            g = w[rows, c] * pre[:, rows, c] + (1 - w[rows, c]) * (
                -self.qx * f[:, rows, n] - self.qtx * o[:, rows, c] - self.qxt * o[:, rows, n])
            f[:, rows, c] = g
        side = f.clone() if not self.fs else f  # the top corners read the sides as they are now
        # bottom: the row above is final; corners also take the x neighbour
        R, U = slice(j0, nz - 1), slice(j0 - 1, nz - 2)
        wb = w[R]
        z = -self.qtz * o[:, R] - self.qxt * o[:, U]
        cols, Pc, Pe = self.P[key]
        mid = slice(b + 1, nx - b - 1)
        A = wb[:, mid] * pre[:, R, mid] + (1 - wb[:, mid]) * z[:, :, mid]
        f[:, R, mid] = torch.einsum("jk,ski->sji", Pe, torch.cat([f[:, j0 - 1:j0, mid], A], 1))

        def corners(cols, nb, take):
            fx = take[:, R][:, :, nb]
            sx = -self.qx * fx - self.qtx * o[:, R][:, :, cols] - self.qxt * o[:, R][:, :, nb]
            A = wb[:, cols] * pre[:, R][:, :, cols] + (1 - wb[:, cols]) * 0.5 * (sx + z[:, :, cols])
            at = torch.searchsorted(self.P[key][0], cols)
            f[:, R, cols] = torch.einsum("ijk,ski->sji", Pc[at], torch.cat([f[:, j0 - 1:j0][:, :, cols], A], 1))

        dev = f.device
        left, right = torch.arange(1, b + 1, device=dev), torch.arange(r0, nx - 1, device=dev)
        first = (right - r0) % 8 == 0
        corners(left[:-1], left[:-1] + 1, pre)
        corners(left[-1:], left[-1:] + 1, f)
        if (~first).any():
            corners(right[~first], right[~first] - 1, pre)
        corners(right[first], right[first] - 1, f)
        if not self.fs:
            T, D = slice(1, b + 1), slice(2, b + 2)
            f[:, T, mid] = self.edge(pre, o, w, (T, mid), (D, mid), self.qz, self.qtz)

            def top(cols, nb, take):
                sx = -self.qx * take[:, T][:, :, nb] - self.qtx * o[:, T][:, :, cols] - self.qxt * o[:, T][:, :, nb]
                sz = -self.qz * side[:, D][:, :, cols] - self.qtz * o[:, T][:, :, cols] - self.qxt * o[:, D][:, :, cols]
                f[:, T, cols] = w[T][:, cols] * side[:, T][:, :, cols] + (1 - w[T][:, cols]) * 0.5 * (sx + sz)

            top(left[:-1], left[:-1] + 1, side)
            top(left[-1:], left[-1:] + 1, f)
            if (~first).any():
                top(right[~first], right[~first] - 1, side)
            top(right[first], right[first] - 1, f)
        return f

    def step(self, k):
        f, M, nx, nz = self.f, self.M, self.nx, self.nz
        I = (slice(None), slice(M, nz - M), slice(M, nx - M))
        J = I[1:]
        old = dict(f)
        xx, zz = f["xx"].clone(), f["zz"].clone()
        for t in (xx, zz):
            t[self.S, self.sj, self.si] += self.wav[k]
        vx, vz, xz = f["vx"].clone(), f["vz"].clone(), f["xz"]
        vx[I] += (self.dtx * self.diff(xx, 2, 0) + self.dtz * self.diff(xz, 1, 0)) / self.rx[J]
        vz[I] += (self.dtx * self.diff(xz, 2, 1) + self.dtz * self.diff(zz, 1, 1)) / self.rz[J]
        f["vx"], f["vz"] = vx, vz = self.habc(vx, old["vx"], "vx"), self.habc(vz, old["vz"], "vz")
        ex, ez = self.dtx * self.diff(vx, 2, 1), self.dtz * self.diff(vz, 1, 0)
        lam, l2m, xz = self.lam[J], (self.lam + 2 * self.mu)[J], xz.clone()
        xx[I] += l2m * ex + lam * ez
        zz[I] += lam * ex + l2m * ez
        xz[I] += self.mxz[J] * (self.dtz * self.diff(vx, 1, 1) + self.dtx * self.diff(vz, 2, 0))
        for name, t in (("xx", xx), ("zz", zz), ("xz", xz)):
            f[name] = self.habc(t, old[name], "t")
        if self.fs:
            rows = slice(max(0, self.pad - 5), self.pad + 1)
            f["zz"][:, rows] = 0.0
            f["xz"][:, rows] = 0.0

    def record(self):
        at = (self.S[:, None], self.rj, self.ri)
        if self.kind == "p":
            return 0.5 * (self.f["xx"][at] + self.f["zz"][at])
        return self.f[self.kind][at]


def _exact_shots(d, jobs, skip=0, downsample=1):
    """Gathers (shot, nt, receiver) of shots with the same nt and receiver count, and frames of p."""
    e = _Exact(d, jobs)
    rows, frames = [], []
    for k in range(jobs[0]["nt"]):
        e.step(k)
        rows.append(e.record())
        if skip and (k + 1) % skip == 0:
            p = 0.5 * (e.f["xx"][0] + e.f["zz"][0])
            frames.append(p[::downsample, ::downsample].T.cpu().numpy())
    return torch.stack(rows, 1).cpu().numpy(), frames


def exact(case, seed):
    grids, shots = _grids(case)
    # about 0.3 ns a cell-step on a GPU, and 2 ms a step (its launches) for each call below
    runs = len(shots) if case["kind"] == "serve" else 1
    cost = sum(3.0e-10 * 1.7 * grids[g][0] * grids[g][1] * nt for g, nt, _ in shots) + 2.5e-3 * runs * case["nt"]
    if cost > 12.0:
        return None
    media, jobs = _survey(case, seed)
    if case["kind"] == "serve":
        return {"gathers": [_exact_shots(media[j["medium"]], [j])[0][0] for j in jobs]}
    if case["kind"] == "batch":
        for j in jobs[1:]:
            j.update(wavelet=jobs[0]["wavelet"])
        return {"gathers": list(_exact_shots(media[0], jobs)[0])}
    g, frames = _exact_shots(media[0], jobs, case.get("skip", 0), case.get("downsample", 1))
    return {"gather": g[0], "frames": np.stack(frames)} if frames else {"gather": g[0]}
