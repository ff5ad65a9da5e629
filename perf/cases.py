"""Performance cases of taichirtm_b200: the work its users have it do.

Each case is one pass through a public entry point, on seeded layered models
with Gaussian anomalies, Ricker sources and hyperbolic-event records.  Kinds:

  run       ReverseTimeMigration().set_...().run() on host arrays: one shot,
            three components, everything the call does (grid, plans, copies).
  shot      ForwardModeling.run(save=True) and BackwardModeling.run_calc() on
            objects the program keeps: the reference's own classes, one shot on
            the whole grid, with their default launch settings.
  model     ForwardModeling.run() alone: seismograms of one shot.
  migrate   BatchedRTM.migrate(): many windowed shots of one model, snapshots
            or 16/32-bit checkpoints, plain or source-normalised imaging.
  gradient  l2_misfit(...).backward() of an FWIProblem: forward modelling and
            the exact adjoint, gradients of vp, vs and rho.

``exact`` restates forward modelling, backward propagation, imaging and (by
autograd) the gradient in float64 torch operations, one shot at a time.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

from taichirtm_b200 import BackwardModeling, ForwardModeling, ReverseTimeMigration
from taichirtm_b200.batch import BatchedRTM
from taichirtm_b200.fwi import FWIProblem, l2_misfit
from taichirtm_b200.plan import ShotGeometry

MODES = {"psv": 1, "sh": 2, "both": 3}


def listed():
    return [
        # the smallest call: seismograms of a test-sized model, both wave types
        dict(name="model_72x56_both", kind="model", nx=72, nz=56, nt=120, fw=8, mode="both", surface=False),
        # one shot of a shallow survey, an image from every time step
        dict(name="shot_301x151_psv", kind="shot", nx=301, nz=151, nt=500, fw=50, mode="psv", surface=False, isnap=1),
        # SH waves, a longer line, snapshots at intervals
        dict(name="shot_1001x501_sh", kind="shot", nx=1001, nz=501, nt=400, fw=50, mode="sh", surface=False, isnap=7),
        # three components under topography, odd sizes
        dict(name="shot_403x207_both_topo", kind="shot", nx=403, nz=207, nt=300, fw=40, mode="both", surface=True,
             isnap=5),
        # the reference's one-call migration from host arrays
        dict(name="run_3c", kind="run", receivers=48, spacing=2.0, velocity=180.0, nt=300, fw=40),
        # one windowed shot of a production line by itself
        dict(name="migrate_1_2001x801", kind="migrate", nx=2001, nz=801, nt=400, fw=50, mode="psv", shots=1, rec_lo=480,
             rec_hi=480, isnap=16, store="snapshots", normalized=False, surface=False),
        # the production batch: 64 windowed shots of that line
        dict(name="migrate_64_2001x801", kind="migrate", nx=2001, nz=801, nt=600, fw=50, mode="psv", shots=64,
             rec_lo=200, rec_hi=800, isnap=16, store="snapshots", normalized=False, surface=False),
        # the same line with compressed checkpoints instead of snapshots
        dict(name="migrate_16_ckpt_i16", kind="migrate", nx=2001, nz=801, nt=500, fw=50, mode="psv", shots=16,
             rec_lo=200, rec_hi=800, isnap=16, store="i16", normalized=False, surface=False),
        # large windows on a deep model, which need checkpoints
        dict(name="migrate_3_4001x1601_ckpt", kind="migrate", nx=4001, nz=1601, nt=200, fw=50, mode="psv", shots=3,
             rec_lo=1000, rec_hi=2000, isnap=16, store="i16", normalized=False, surface=False),
        # source-normalised imaging of SH shots under topography
        dict(name="migrate_8_sh_normalized", kind="migrate", nx=801, nz=301, nt=400, fw=40, mode="sh", shots=8,
             rec_lo=150, rec_hi=400, isnap=10, store="snapshots", normalized=True, surface=True),
        # the gradient of a multi-shot inversion, launch shape tuned as its benchmark does
        dict(name="gradient_8_1201x401", kind="gradient", nx=1201, nz=401, nt=500, fw=50, shots=8, store="f32",
             tuned=True, double=True),
        # a small inversion on the default launch shape
        dict(name="gradient_1_201x101", kind="gradient", nx=201, nz=101, nt=300, fw=20, shots=1, store="f32",
             tuned=False, double=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, sizes over their whole ranges."""
    kind = rng.choice(["model", "shot", "shot", "run", "migrate", "migrate", "migrate", "gradient"])
    if kind == "run":
        return dict(kind=kind, receivers=rng.randint(12, 96), spacing=round(rng.uniform(1.0, 3.0), 2),
                    velocity=round(rng.uniform(120.0, 300.0), 1), nt=_log(rng, 100, 500), fw=rng.randint(20, 60))
    if kind in ("model", "shot"):
        nx, nz = _log(rng, 48, 1001), _log(rng, 40, 501)
        c = dict(kind=kind, nx=nx, nz=nz, nt=_log(rng, 60, 600), fw=rng.randint(4, max(5, min(60, nx // 3, nz // 3))),
                 mode=rng.choice(["psv", "psv", "sh", "both"]), surface=rng.random() < 0.3)
        if kind == "shot":
            c["isnap"] = _log(rng, 1, 20)
        return c
    if kind == "migrate":
        nx, nz = _log(rng, 301, 2401), _log(rng, 151, 1201)
        hi = max(60, min(800, nx // 2))
        lo = rng.randint(40, hi)
        store = rng.choice(["snapshots", "snapshots", "snapshots", "i16", "f16", "bf16", "f32"])
        mode = "psv" if store != "snapshots" else rng.choice(["psv", "psv", "sh", "both"])
        nt = _log(rng, 100, 600)
        most = max(1, int(28e6 * 600 / 2 / ((hi + 100) * nz * nt)))  # at most half the largest listed batch
        return dict(kind=kind, nx=nx, nz=nz, nt=nt, fw=rng.randint(20, 50), mode=mode,
                    shots=_log(rng, 1, min(64, most)), rec_lo=lo, rec_hi=hi, isnap=_log(rng, 4, 20), store=store,
                    normalized=store == "snapshots" and rng.random() < 0.25, surface=rng.random() < 0.25)
    nx, nz = _log(rng, 101, 1201), _log(rng, 61, 401)
    return dict(kind=kind, nx=nx, nz=nz, nt=_log(rng, 100, 500), fw=rng.randint(10, max(11, min(50, nx // 3, nz // 3))),
                shots=_log(rng, 1, 8), store=rng.choice(["f32", "f32", "i16", "f16"]), tuned=rng.random() < 0.5,
                double=rng.random() < 0.5)


# --------------------------------------------------------------------- inputs
DX, FS = 5.0, 2000.0  # grid step (m) and sampling rate (Hz) of every kind but "run"


def _geometry(case):
    """Sizes that follow from the case alone: per shot (x0, nx, source, receivers)."""
    if case["kind"] != "migrate":
        n = case.get("shots", 1)
        nx = case["nx"]
        out = []
        for k in range(n):
            c = nx // 2 if n == 1 else int(round(nx * (0.15 + 0.7 * k / (n - 1))))
            rec = np.stack([np.arange(nx), np.ones(nx, int)], 1)
            out.append((0, nx, np.array([[c, 2]]), rec))
        return out
    n, nx, fw = case["shots"], case["nx"], case["fw"]
    out = []
    for k in range(n):
        c = nx // 2 if n == 1 else int(round(fw + (nx - 1 - 2 * fw) * k / (n - 1)))
        cnt = case["rec_lo"] + (k * 7919) % (case["rec_hi"] - case["rec_lo"] + 1)
        r0 = min(max(0, c - cnt // 2), nx - 1)
        r1 = min(nx, r0 + cnt)
        x0, x1 = max(0, min(r0, c) - fw), min(nx, max(r1, c + 1) + fw)
        rec = np.stack([np.arange(r0, r1) - x0, np.ones(r1 - r0, int)], 1)
        out.append((x0, x1 - x0, np.array([[c - x0, 2]]), rec))
    return out


def _ricker(t, f):
    a = (math.pi * f * (t - 1.0 / f)) ** 2
    return (1.0 - 2.0 * a) * torch.exp(-a)


def _model(nx, nz, gen, dev, smooth=False):
    """(vp, vs, rho) float64: four layers and seeded anomalies; smooth: their low-contrast version."""
    z = torch.arange(nz, dtype=torch.float64, device=dev)
    x = torch.arange(nx, dtype=torch.float64, device=dev)
    speeds = (1500.0, 2200.0, 2900.0, 3500.0)
    prof = torch.full((nz,), speeds[0], dtype=torch.float64, device=dev)
    w = max(1.0, nz / 25.0) if smooth else 0.5
    for k in range(3):
        prof = prof + (speeds[k + 1] - speeds[k]) * torch.sigmoid((z - nz * (k + 1) / 4.0) / w)
    vp = prof.expand(nx, nz).clone()
    for _ in range(12):
        cx, cz, a, s = torch.rand(4, generator=gen, dtype=torch.float64).tolist()
        s = 8.0 + 30.0 * s
        g = torch.exp(-((x - cx * nx) ** 2) / (2 * s * s))[:, None] * torch.exp(-((z - cz * nz) ** 2) / (2 * s * s))
        vp = vp * (1.0 + (0.24 * a - 0.12) * g * (0.4 if smooth else 1.0))
    return vp, vp / 1.73, 310.0 * vp ** 0.25


def _lame(vp, vs, rho):
    mu = rho * vs * vs
    return mu.float(), (rho * vp * vp - 2.0 * mu).float(), rho.float()


def _records(offsets, nt, dt, freq, velocity, gen, dev):
    """(3, nrec, nt) float32: a direct arrival, three reflections and a little noise."""
    t = torch.arange(nt, dtype=torch.float64, device=dev) * dt
    x = torch.as_tensor(offsets, dtype=torch.float64, device=dev)[:, None]
    out = torch.zeros((3, x.shape[0], nt), dtype=torch.float64, device=dev)
    for k in range(4):
        a = torch.rand(4, generator=gen, dtype=torch.float64).tolist()
        t0 = 0.0 if k == 0 else nt * dt * (0.15 + 0.2 * k * (0.7 + 0.6 * a[3]) / 1.3)
        arr = torch.sqrt(t0 ** 2 + (x / (velocity * (1.0 + 0.25 * k))) ** 2)
        amp = (1.0 + k) ** -1 / (1.0 + 0.01 * x.abs())
        for c in range(3):
            out[c] += (0.4 + a[c]) * amp * _ricker(t[None] - arr, freq)
    noise = torch.randn((3, x.shape[0], nt), generator=gen, dtype=torch.float32).to(dev).double()
    return (1e-9 * (out + 0.01 * noise)).float()


def _mask(case, gen, dev):
    """0/1 topography mask: air above a smooth surface a few cells deep (the receiver row stays solid)."""
    nx, nz = case["nx"], case["nz"]
    x = torch.arange(nx, dtype=torch.float64, device=dev)
    a, b = torch.rand(2, generator=gen, dtype=torch.float64).tolist()
    depth = (0.5 + 0.5 * torch.sin(2 * math.pi * (x / nx * (1.0 + 2.0 * a) + b))).round()
    return (torch.arange(nz, device=dev)[None] >= depth[:, None]).float()


def _inputs(case, seed, dev):
    """Everything that the seed decides, on ``dev``."""
    gen = torch.Generator().manual_seed(int(seed) * 1000003 + case["nt"])
    if case["kind"] == "run":
        n, nt, v = case["receivers"], case["nt"], case["velocity"]
        fs = 20.0 * v / (0.4 * case["spacing"] * 4.0)  # a few cells per receiver
        loc = np.arange(n, dtype=np.float32) * np.float32(case["spacing"])
        src = float(loc[n // 3])
        dt = 1.0 / fs
        obs = _records(loc - src, nt, dt, fs / 30.0, v, gen, torch.device("cpu")).numpy()
        w = _ricker(torch.arange(nt, dtype=torch.float64) * dt, fs / 30.0).float().numpy()
        amp = (0.5 + torch.rand(3, generator=gen)).numpy()
        return dict(fs=fs, loc=loc, src=src, obs=obs, wav=[np.float32(a) * w for a in amp])
    geo = _geometry(case)
    nt, dt = case["nt"], 1.0 / FS
    mode = case.get("mode", "psv")
    freq = 25.0 if nt >= 200 else 60.0
    vp, vs, rho = _model(case["nx"], case["nz"], gen, dev, smooth=case["kind"] in ("migrate", "gradient"))
    t = torch.arange(nt, dtype=torch.float64, device=dev) * dt
    wav = torch.zeros((3, len(geo), nt), dtype=torch.float32, device=dev)
    for c in range(3):
        if (c == 1) == (mode == "sh") or mode == "both":
            for s in range(len(geo)):
                wav[c, s] = ((0.5 + float(torch.rand(1, generator=gen))) * _ricker(t, freq)).float()
    obs = torch.cat([_records((r[:, 0] - s[0, 0]) * DX, nt, dt, freq, 1500.0, gen, dev) for _, _, s, r in geo], 1)
    if mode == "psv":
        obs[1] = 0
    elif mode == "sh":
        obs[0] = 0
        obs[2] = 0
    surf = _mask(case, gen, dev) if case.get("surface") else None
    return dict(geo=geo, vp=vp, vs=vs, rho=rho, wav=wav, obs=obs, surface=surf)


# ---------------------------------------------------------------- the passes
def _fields(case, d):
    mu, lam, rho = _lame(d["vp"], d["vs"], d["rho"])
    _, nx, src, rec = d["geo"][0]
    return dict(nx=nx, nz=case["nz"], dx=DX, dz=DX, nt=case["nt"], fs=FS, absorbing_frame=case["fw"], mu_field=mu,
                lam_field=lam, rho_field=rho, src_loc_field=src.astype(np.int32),
                recv_loc_field=rec.astype(np.int32), surface_matrix_field=d["surface"], num_sources=len(src),
                num_receivers=len(rec))


def prepare(case, seed):
    dev = torch.device("cuda")
    d = _inputs(case, seed, dev)
    kind = case["kind"]
    st = dict(case=case, d=d)
    if kind in ("model", "shot"):
        w, f = d["wav"], _fields(case, d)
        st["fm"] = ForwardModeling(wavelet_u_field=w[0], wavelet_v_field=w[1], wavelet_w_field=w[2],
                                   isnap=case.get("isnap", 10), **f)
        if kind == "shot":
            o = d["obs"]
            st["bm"] = BackwardModeling(obsdata_u_field=o[0], obsdata_v_field=o[1], obsdata_w_field=o[2], **f)
    elif kind == "migrate":
        shots = [ShotGeometry(*g) for g in d["geo"]]
        st["rtm"] = BatchedRTM(*_lame(d["vp"], d["vs"], d["rho"]), DX, DX, FS, case["nt"], case["fw"], shots,
                               modes=MODES[case["mode"]], surface=d["surface"])
    elif kind == "gradient":
        shots = [ShotGeometry(*g) for g in d["geo"]]
        st["problem"] = FWIProblem(case["nx"], case["nz"], DX, DX, FS, case["nt"], case["fw"], shots, d["wav"],
                                   tune="auto" if case["tuned"] else None, ckpt_dtype=case["store"])
        st["m"] = [(x if case["double"] else x.float()) for x in (d["vp"], d["vs"], d["rho"])]
    return st


def run(st):
    case, d, kind = st["case"], st["d"], st["case"]["kind"]
    if kind == "model":
        flag = st["fm"].run()
        return dict(flag=flag, seis=st["fm"].get_seismogram_tensors())
    if kind == "shot":
        fm, bm = st["fm"], st["bm"]
        flag = fm.run(save=True)
        back = bm.run_calc(fm.u_save_field, fm.v_save_field, fm.w_save_field, fm.isnaps_field, fm.num_snaps,
                           case["isnap"])
        return dict(flag=flag, back=back, seis=fm.get_seismogram_tensors(), image=bm.get_result_tensors())
    if kind == "run":
        with ReverseTimeMigration() as rtm:
            rtm.set_observed_data(*d["obs"]).set_source(*d["wav"], d["src"]).set_receivers(d["loc"])
            rtm.set_frequency(d["fs"]).fix_velocity(case["velocity"]).set_boundary(case["fw"])
            rtm.set_poisson_ratio(0.2).run()
            return dict(image=np.stack(rtm.get_results()))
    if kind == "migrate":
        ck = None if case["store"] == "snapshots" else dict(every=None, dtype=case["store"])
        method = "source_normalized" if case["normalized"] else "cross_correlation"
        ff, fb, stack = st["rtm"].migrate(d["wav"], d["obs"], isnap=case["isnap"], checkpoint=ck, method=method)
        return dict(forward_flags=ff, backward_flags=fb, image=stack)
    m = [x.clone().requires_grad_(True) for x in st["m"]]
    J = l2_misfit(m[0], m[1], m[2], st["problem"], d["obs"])
    J.backward()
    return dict(misfit=J.detach(), grads=[x.grad for x in m])


# ------------------------------------------------------------------ the floor
def _cells(case):
    if case["kind"] == "run":
        n = int((case["receivers"] - 1) * case["spacing"] / _run_dx(case)) + 4 * case["fw"]
        return n * n, n * n
    geo = _geometry(case)
    rows = set()
    for x0, nx, _, _ in geo:
        rows.update(range(x0, x0 + nx))
    return sum(g[1] for g in geo) * case["nz"], len(rows) * case["nz"]


def _run_dx(case):
    fs = 20.0 * case["velocity"] / (0.4 * case["spacing"] * 4.0)
    return case["velocity"] / fs / 0.4


# additions and multiplications of one cell and time step
STEP_FLOPS = {"psv": 39, "sh": 18, "both": 57}
ADJOINT_FLOPS = 96


def work(case):
    """Inputs read and outputs written once; the stencils' operations."""
    cells, model = _cells(case)
    nt = case["nt"]
    nrec = case["receivers"] if case["kind"] == "run" else sum(len(g[3]) for g in _geometry(case))
    traces = 12 * nrec * nt
    per = STEP_FLOPS[case.get("mode", "both" if case["kind"] == "run" else "psv")]
    if case["kind"] == "model":
        return dict(bytes=12 * model + traces, flops=cells * nt * per)
    if case["kind"] == "gradient":
        w = 8 if case["double"] else 4
        return dict(bytes=2 * 3 * w * model + traces, flops=cells * nt * (per + ADJOINT_FLOPS))
    out = 24 * model if case["kind"] == "migrate" else 12 * model + traces
    return dict(bytes=12 * model + traces + out, flops=2 * cells * nt * per)


# ------------------------------------------------- the same values in 64 bits
def _pad(x):
    return torch.nn.functional.pad(x, (1, 1, 1, 1))


class _Exact:
    """Float64 steps of one shot on its window (coefficients zero on the edges, where nothing is updated)."""

    def __init__(self, mu, lam, rho, dx, fs, fw, surface=None):
        self.dx, self.dt = dx, 1.0 / fs
        nx, nz = mu.shape
        a, b, c, d = mu[1:-1, 1:-1], mu[2:, 1:-1], mu[1:-1, 2:], mu[2:, 2:]
        self.myx, self.myz = 2 * a * b / (a + b), 2 * a * c / (a + c)
        self.mxz = 4 / (1 / a + 1 / b + 1 / c + 1 / d)
        r = rho[1:-1, 1:-1]
        self.bu, self.bw, self.bv = 2 / (r + rho[2:, 1:-1]), 2 / (r + rho[1:-1, 2:]), 1 / r
        self.lam, self.mu = lam[1:-1, 1:-1], a
        i = torch.arange(nx, device=mu.device)[:, None].expand(nx, nz)
        j = torch.arange(nz, device=mu.device)[None].expand(nx, nz)
        dr, db = nx - 1 - i, nz - 1 - j
        dist = torch.full_like(i, fw)
        dist = torch.where((i < fw) & (db > i), i, dist)
        dist = torch.where((dr < fw) & (db > dr), dr, dist)
        dist = torch.where((db < fw) & (i >= db) & (dr >= db), db, dist)
        self.c = torch.exp(-((0.0053 * (fw - dist).double()) ** 2))
        self.m = torch.ones_like(mu) if surface is None else surface

    def zero(self):
        return tuple(torch.zeros_like(self.c) for _ in range(8))

    def absorb(self, v, s):
        c, cm = self.c, self.c * self.m
        return (v[0] * c, v[1] * c, v[2] * c, s[0] * c, s[1] * cm, s[2] * cm, s[3] * c, s[4] * cm)

    def forward(self, st, src, wav, psv=True, sh=True):
        u, v, w, xx, zz, xz, yx, yz = st
        h, dt = 1.0 / self.dx, self.dt
        I, up, lf, dn, rt = ((slice(1, -1), slice(1, -1)), (slice(None, -2), slice(1, -1)),
                             (slice(1, -1), slice(None, -2)), (slice(2, None), slice(1, -1)),
                             (slice(1, -1), slice(2, None)))
        inj = dt * self.dx * self.dx
        if psv:
            u = u + _pad(((xx[I] - xx[up]) + (xz[I] - xz[lf])) * h * dt * self.bu)
            w = w + _pad(((xz[I] - xz[up]) + (zz[I] - zz[lf])) * h * dt * self.bw)
            for k, (i, j) in enumerate(src):
                e = torch.zeros_like(u)
                e[i, j] = inj
                u = u + e * wav[0, k] * _pad(self.bu)
                w = w + e * wav[2, k] * _pad(self.bw)
            ux, uz = (u[dn] - u[I]) * h, (u[rt] - u[I]) * h
            wx, wz = (w[dn] - w[I]) * h, (w[rt] - w[I]) * h
            xx = xx + _pad(dt * (self.lam * (ux + wz) + 2 * self.mu * ux))
            zz = zz + _pad(dt * (self.lam * (ux + wz) + 2 * self.mu * wz))
            xz = xz + _pad(dt * self.mxz * (uz + wx))
        if sh:
            v = v + _pad(((yx[I] - yx[up]) + (yz[I] - yz[lf])) * h * dt * self.bv)
            for k, (i, j) in enumerate(src):
                e = torch.zeros_like(v)
                e[i, j] = inj
                v = v + e * wav[1, k] * _pad(self.bv)
            yx = yx + _pad(dt * self.myx * (v[dn] - v[I]) * h)
            yz = yz + _pad(dt * self.myz * (v[rt] - v[I]) * h)
        return self.absorb((u, v, w), (xx, zz, xz, yx, yz))

    def backward(self, st, rec, obs, psv=True, sh=True):
        u, v, w, xx, zz, xz, yx, yz = st
        h, dt = 1.0 / self.dx, self.dt
        I, up, lf, dn, rt = ((slice(1, -1), slice(1, -1)), (slice(None, -2), slice(1, -1)),
                             (slice(1, -1), slice(None, -2)), (slice(2, None), slice(1, -1)),
                             (slice(1, -1), slice(2, None)))
        at = (rec[:, 0], rec[:, 1])
        if psv:
            u = u - _pad(((xx[dn] - xx[I]) + (xz[rt] - xz[I])) * h * dt * self.bu)
            w = w - _pad(((xz[dn] - xz[I]) + (zz[rt] - zz[I])) * h * dt * self.bw)
            u = u.index_put(at, obs[0], accumulate=True)
            w = w.index_put(at, obs[2], accumulate=True)
            ux, uz = (u[I] - u[up]) * h, (u[I] - u[lf]) * h
            wx, wz = (w[I] - w[up]) * h, (w[I] - w[lf]) * h
            xx = xx - _pad(dt * (self.lam * (ux + wz) + 2 * self.mu * ux))
            zz = zz - _pad(dt * (self.lam * (ux + wz) + 2 * self.mu * wz))
            xz = xz - _pad(dt * self.mxz * (uz + wx))
        if sh:
            v = v - _pad(((yx[dn] - yx[I]) + (yz[rt] - yz[I])) * h * dt * self.bv)
            v = v.index_put(at, obs[1], accumulate=True)
            yx = yx - _pad(dt * self.myx * (v[I] - v[up]) * h)
            yz = yz - _pad(dt * self.myz * (v[I] - v[lf]) * h)
        return self.absorb((u, v, w), (xx, zz, xz, yx, yz))


def _exact_shot(ex, src, rec, wav, obs, isnap, psv, sh, image=True):
    """(seismograms, image (None without image), illumination) of one shot."""
    nt = wav.shape[2]
    rec = torch.as_tensor(np.asarray(rec, np.int64), device=wav.device)
    seis = torch.zeros((3, len(rec), nt), dtype=torch.float64, device=wav.device)
    st, snaps = ex.zero(), {}
    nsnap = nt // isnap
    for it in range(nt):
        st = ex.forward(st, src, wav[:, :, it], psv, sh)
        for c in range(3):
            seis[c, :, it] = st[c][rec[:, 0], rec[:, 1]]
        if image and it % isnap == 0 and it and it // isnap <= nsnap:
            snaps[it] = tuple(x.clone() for x in st[:3])
    if not image:
        return seis, None, None
    st = ex.zero()
    img = [torch.zeros_like(ex.c) for _ in range(3)]
    ill = [torch.zeros_like(ex.c) for _ in range(3)]
    for t in range(nt - 1, -1, -1):
        st = ex.backward(st, rec, obs[:, :, t], psv, sh)
        if t in snaps:
            for c in range(3):
                img[c] += snaps[t][c] * st[c]
                ill[c] += snaps[t][c] ** 2
    return seis, torch.stack(img), torch.stack(ill)


def _exact_gradient(case, d, dev):
    leaves = [(x if case["double"] else x.float()).double().requires_grad_(True) for x in (d["vp"], d["vs"], d["rho"])]
    vp, vs, rho = leaves
    total = 0.0
    nt, r0 = case["nt"], 0
    K = max(1, round(math.sqrt(nt)))
    for s, (_, _, src, rec) in enumerate(d["geo"]):
        obs = d["obs"][:, r0:r0 + len(rec)].double()
        r0 += len(rec)
        at = torch.as_tensor(rec, device=dev, dtype=torch.int64)
        wav = d["wav"][:, s:s + 1].double()

        def segment(t0, t1, vp, vs, rho, *st):
            mu = rho * vs * vs
            ex = _Exact(mu, rho * vp * vp - 2 * mu, rho, DX, FS, case["fw"])
            st, J = (st[0], ex.zero()[0], *st[1:], ex.zero()[0], ex.zero()[0]), 0.0
            for it in range(t0, t1):
                st = ex.forward(st, src, wav[:, :, it], True, False)
                for c in (0, 2):
                    J = J + 0.5 * ((st[c][at[:, 0], at[:, 1]] - obs[c, :, it]) ** 2).sum()
            return (J, st[0], st[2], st[3], st[4], st[5])

        st = tuple(torch.zeros_like(vp) for _ in range(5))
        J = 0.0
        for t0 in range(0, nt, K):
            part, *st = torch.utils.checkpoint.checkpoint(segment, t0, min(nt, t0 + K), vp, vs, rho, *st,
                                                          use_reentrant=False)
            J = J + part
        J.backward()
        total += float(J.detach())
    return dict(misfit=torch.tensor(total, dtype=torch.float64), grads=[x.grad for x in leaves])


def exact(case, seed):
    cells, _ = _cells(case)
    kind, nt = case["kind"], case["nt"]
    n = case.get("shots", 1)
    # about 70 kernels a step, each a few microseconds or three passes over the window
    step = 70 * max(6e-6, 24.0 * cells / n / 3e12)
    if step * nt * n * (4 if kind == "gradient" else 2) > 15.0:
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    d = _inputs(case, seed, dev)
    if kind == "gradient":
        return _exact_gradient(case, d, dev)
    if kind == "run":
        v, fs, fw = case["velocity"], d["fs"], case["fw"]
        dx = v / fs / 0.4
        size = int((d["loc"].max() - d["loc"].min()) / dx) + 4 * fw
        one = np.ones((size, size), np.float32)
        rho, vs = one * np.float32(1500), one * np.float32(v)
        vp = (np.sqrt((2 * 0.2 + 1) / (1 - 2 * 0.2)) * vs).astype(np.float32)
        mu = (rho * vs ** 2).astype(np.float32)
        lam = (((vp / vs) ** 2 - 2) * mu).astype(np.float32)
        ex = _Exact(*(torch.as_tensor(x, device=dev).double() for x in (mu, lam, rho)), dx, fs, fw)
        rec = np.array([[int(x / dx + 2 * fw), 1] for x in d["loc"]])
        src = np.array([[int(d["src"] / dx + 2 * fw), 1]])
        wav = torch.as_tensor(np.stack(d["wav"])[:, None], device=dev).double()
        _, img, _ = _exact_shot(ex, src, rec, wav, torch.as_tensor(d["obs"], device=dev).double(), 1, True, True)
        return dict(image=img)
    mu, lam, rho = (x.double() for x in _lame(d["vp"], d["vs"], d["rho"]))
    surf = None if d["surface"] is None else d["surface"].double()
    psv, sh = case["mode"] != "sh", case["mode"] != "psv"
    stack = torch.zeros((3,) + tuple(mu.shape), dtype=torch.float64, device=dev)
    r0 = 0
    for s, (x0, nx, src, rec) in enumerate(d["geo"]):
        w = slice(x0, x0 + nx)
        ex = _Exact(mu[w], lam[w], rho[w], DX, FS, case["fw"], None if surf is None else surf[w])
        seis, img, ill = _exact_shot(ex, src, rec, d["wav"][:, s:s + 1].double(),
                                     d["obs"][:, r0:r0 + len(rec)].double(), case.get("isnap", 10), psv, sh,
                                     image=kind != "model")
        r0 += len(rec)
        if kind == "model":
            return dict(flag=None, seis=seis)
        if kind == "shot":
            return dict(flag=None, back=None, seis=seis, image=img)
        if case["normalized"]:
            den = ill + float(np.float32(1e-3)) * ill.amax(dim=(1, 2), keepdim=True)
            img = torch.where(den > 0, img / den, torch.zeros_like(img))
        stack[:, w] += img
    return dict(forward_flags=None, backward_flags=None, image=stack)
