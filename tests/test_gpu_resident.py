"""Resident propagation (plans whose launch shape is the library's choice and
whose wavefield fits on the chip) against the streaming kernels, which other
tests pin to the FP32 restatement: seismograms, snapshots, images, status codes
and the final wavefield are the same floats (tolerance 0), at the sizes where
the tiles end, for every layout, wave type and kind of point entry."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
STREAM = dict(vec=2, rows=5, warps=2, tsteps=1)


def _model(nx, nz, seed=1):
    rng = np.random.default_rng(seed)
    vp = 2000.0 + 600.0 * rng.random((nx, nz))
    vs, rho = vp / 1.8, 310.0 * vp ** 0.25
    mu = (rho * vs ** 2).astype(np.float32)
    return mu, (rho * vp ** 2).astype(np.float32) - 2 * mu, rho.astype(np.float32)


def _points(nx, nz, dense):
    """Sources (two in one cell, one beside it, one on the edge column) and
    receivers: a line, and if dense whole rows, duplicates and edge cells."""
    src = np.array([[nx // 2, nz // 2], [nx // 2, nz // 2], [nx // 2, min(nz // 2 + 1, nz - 2)], [1, 1]], np.int32)
    rec = [[i, min(1, nz - 1)] for i in range(nx)]
    if dense:
        rec += [[nx // 2, j] for j in range(nz)] + [[0, 0], [nx - 1, nz - 1], [nx // 2, 1], [nx // 2, 1]]
    return src, np.array(rec, np.int32)


def _run(shots, nx, nz, nt, fw, modes, tune, wav, isnap, check, surface=None, resident=None, obs=None):
    from taichirtm_b200.plan import Plan
    p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, fw, modes, shots, tune=tune)
    p.set_model(*_model(nx, nz), surface)
    assert resident is None or p.resident() == resident
    out = []
    f, seis, snaps, isn = p.forward(torch.as_tensor(wav), save=True, isnap=isnap, check_interval=check)
    out += [f, seis.cpu().numpy()]
    if f.max() == 0:  # a stopped shot's last wavefield lies one step apart in the two
        out += [p.wavefield(s).cpu().numpy() for s in range(len(shots))]
    for s in range(len(shots)):
        if f[s] == 0:
            out += [p.snapshot_view(b, len(isn), s).cpu().numpy() for b in snaps if b is not None]
    o = torch.as_tensor(np.nan_to_num(out[1], nan=0.5, posinf=0.5, neginf=0.5) * 0.5 + np.float32(1e-3)) if obs is None else obs
    stack = torch.zeros((3, nx, nz), dtype=torch.float64, device="cuda")
    for b in snaps:
        if b is not None:
            torch.nan_to_num_(b, nan=0.0, posinf=0.0, neginf=0.0)
    fb, _, _ = p.backward(o, snaps, isn, len(isn), isnap, check_interval=check, image=False, stack=stack)
    out += [fb, stack.cpu().numpy()]
    p.close()
    return out


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")


def _wavelets(n, nt, seed=3):
    w = np.random.default_rng(seed).standard_normal((3, n, nt)).astype(np.float32)
    w[:, :, nt // 2:] = 0
    return w


# widths around the 56 columns and heights around the 8, 16 and 40 rows that a
# tile owns, the smallest grid, and steps around the 4 between exchanges
@pytest.mark.parametrize("modes", [1, 2, 3])
@pytest.mark.parametrize("grid,nt,isnap", [((3, 3), 5, 1), ((7, 55), 4, 1), ((8, 56), 1, 1), ((9, 57), 9, 2),
                                           ((17, 113), 13, 3), ((41, 60), 8, 4)])
def test_tile_edges(grid, nt, isnap, modes):
    from taichirtm_b200.plan import ShotGeometry
    nx, nz = grid
    src, rec = _points(nx, nz, dense=nx > 8)
    shots = [ShotGeometry(0, nx, src[:1] if nx == 3 else src, rec)]
    wav = _wavelets(len(shots[0].src), nt)
    for fw, check in ((0, 0), (min(nx, nz) // 3, 3)):
        a = _run(shots, nx, nz, nt, fw, modes, None, wav, isnap, check, resident=True)
        _same(a, _run(shots, nx, nz, nt, fw, modes, STREAM, wav, isnap, check, resident=False))
    assert nt == 1 or np.abs(a[1]).max() > 0  # one step: the wavelets are zero from nt // 2 on


# one shot per layout: the sizes at which the others are estimated slower
@pytest.mark.parametrize("modes,grid", [(1, (300, 150)), (1, (400, 250)), (1, (560, 700)), (2, (400, 251)), (2, (610, 420)),
                                        (2, (900, 800)), (3, (200, 100)), (3, (300, 300)), (3, (431, 417))])
@pytest.mark.parametrize("topography", [False, True])
def test_every_layout(modes, grid, topography):
    from taichirtm_b200.plan import ShotGeometry
    nx, nz = grid
    surface = None
    if topography:  # a mask with fractions, too
        surface = np.ones((nx, nz), np.float32)
        surface[: nx // 2, :2] = 0
        surface[nx // 2: nx // 2 + 9, 3] = 0.25
    src, rec = _points(nx, nz, dense=False)
    shots = [ShotGeometry(0, nx, src, rec)]
    wav = _wavelets(len(src), 14)
    a = _run(shots, nx, nz, 14, 30, modes, None, wav, 5, 6, surface)
    _same(a, _run(shots, nx, nz, 14, 30, modes, STREAM, wav, 5, 6, surface))


def test_windows_in_several_launches():
    """Windowed shots, more than one launch holds, of different sizes."""
    from taichirtm_b200.plan import ShotGeometry
    nx, nz, nt = 700, 330, 11
    shots = []
    for k in range(30):
        w = 120 + 37 * k % 200
        src, rec = _points(w, nz, dense=k % 3 == 0)
        shots.append(ShotGeometry((41 * k) % (nx - w), w, src, rec))
    wav = _wavelets(sum(len(s.src) for s in shots), nt)
    a = _run(shots, nx, nz, nt, 20, 2, None, wav, 4, 5, resident=True)
    _same(a, _run(shots, nx, nz, nt, 20, 2, STREAM, wav, 4, 5))


@pytest.mark.parametrize("check", [1, 2, 3, 5, 7])
def test_failing_shots_stop_at_the_same_check(check):
    """A source on an edge cell injects inf; the other shot goes on."""
    from taichirtm_b200.plan import ShotGeometry
    nx, nz, nt = 190, 130, 23
    _, rec = _points(120, nz, dense=True)
    shots = [ShotGeometry(0, 120, np.array([[0, 30]], np.int32), rec),
             ShotGeometry(70, 120, np.array([[60, 30]], np.int32), rec)]
    wav = _wavelets(2, nt)
    wav[:, :, :4] = 0
    a = _run(shots, nx, nz, nt, 10, 3, None, wav, 2, check, resident=True)
    assert a[0][0] > 0 and a[0][1] == 0
    _same(a, _run(shots, nx, nz, nt, 10, 3, STREAM, wav, 2, check))


@pytest.mark.parametrize("store", ["f32", "f16", "bf16", "i16"])
@pytest.mark.parametrize("every,nt,isnap,check", [(1, 7, 2, 0), (5, 23, 1, 4), (8, 24, 3, 8), (40, 23, 4, 5)])
@pytest.mark.parametrize("windows,nz", [(((0, 121), (99, 131)), 131), (((45, 75),), 101)])
def test_checkpointed_segments(store, every, nt, isnap, check, windows, nz):
    """Checkpoint slots, seismograms and the image of checkpointed RTM, and the
    gradient from those checkpoints, equal the streaming kernels' (vec 2).  The
    single window's state is no multiple of 256 bytes, the slots' alignment."""
    import ctypes
    from taichirtm_b200 import _lib
    from taichirtm_b200.plan import Plan, ShotGeometry, _i32p, _ptr, _stream, check as ok
    nx, fw = 230, 12
    shots = [ShotGeometry(x0, n, *_points(n, nz, dense=x0 == 0)) for x0, n in windows]
    wav = torch.as_tensor(_wavelets(sum(len(s.src) for s in shots), nt)).cuda()
    L, dt, res = _lib.lib(), _lib.CKPT_DTYPES[store], []
    for tune in (None, dict(vec=2, rows=9, warps=2, tsteps=2)):
        p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, fw, 1, shots, tune=tune)
        p.set_model(*_model(nx, nz))
        assert p.resident() == (tune is None)
        ck = torch.zeros(max(int(L.rtm_plan_checkpoint_bytes(p.h, every, dt)), 1), dtype=torch.uint8, device="cuda")
        seis = torch.zeros((3, p.nrec_total, nt), device="cuda")
        stack = torch.zeros((3, nx, nz), dtype=torch.float64, device="cuda")
        grad = torch.zeros((5, nx, nz), dtype=torch.float64, device="cuda")
        flags, flags_b = np.zeros(len(shots), np.int32), np.zeros(len(shots), np.int32)
        ok(L.rtm_forward_checkpointed(p.h, _ptr(wav), _ptr(seis), every, dt, _ptr(ck), check, _i32p(flags), _stream()), "f")
        obs = (seis * 0.5 + 1e-3).contiguous()
        ok(L.rtm_backward_checkpointed(p.h, _ptr(wav), _ptr(obs), every, dt, _ptr(ck), isnap, None, _ptr(stack), check,
                                       _i32p(flags_b), _stream()), "b")
        ok(L.rtm_adjoint(p.h, _ptr(wav), _ptr(obs), every, dt, _ptr(ck), _ptr(grad), ctypes.c_void_p(0), _stream()), "a")
        # FP32 slots are compared through the image and the gradient read from them
        res.append([flags, flags_b] + [x.cpu().numpy() for x in (seis, stack, grad)] + ([ck.cpu().numpy()] if dt else []))
        p.close()
    assert np.abs(res[0][3]).max() > 0 and np.abs(res[0][4]).max() > 0
    _same(*res)


def test_two_threads_and_streams():
    """Two plans propagate at the same time, each in a host thread and on a
    stream of its own; together they ask for more tiles than the chip holds."""
    import threading
    from taichirtm_b200.plan import Plan, ShotGeometry
    nx, nz, nt = 300, 400, 200
    src, rec = _points(nx, nz, dense=False)
    wav = torch.as_tensor(_wavelets(len(src), nt)).cuda()
    plans = []
    for _ in range(2):
        p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 20, 1, [ShotGeometry(0, nx, src, rec)])
        p.set_model(*_model(nx, nz))
        assert p.resident()
        plans.append(p)
    want = plans[0].forward(wav)[1].clone()
    torch.cuda.synchronize()
    same, errors = [], []

    def work(p, stream):
        try:
            for _ in range(10):
                flags, seis, _, _ = p.forward(wav, stream=stream)  # returns after the stream's work
                same.append(flags[0] == 0 and torch.equal(seis, want))
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)
    threads = [threading.Thread(target=work, args=(p, torch.cuda.Stream())) for p in plans]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    for p in plans:
        p.close()
    assert not errors and len(same) == 20 and all(same)
