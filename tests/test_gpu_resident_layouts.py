"""Every tile layout of the resident loops by name, and their less frequent paths,
against the streaming kernels (tolerance 0)."""
import ctypes

import numpy as np
import pytest
import torch

from tests.test_gpu_resident import STREAM, _model, _points, _run, _same, _wavelets

pytestmark = pytest.mark.gpu


def _layout(nx, nz, modes, shots, surface=None):
    from taichirtm_b200.plan import Plan
    p = Plan(nx, nz, 4.0, 4.0, 8, 2000.0, 4, modes, shots)
    p.set_model(*_model(nx, nz), surface)
    got = p.resident_layout()
    p.close()
    return got


# rows per lane of the P-SV and SH tiles, warps; a grid on which it is the fastest by
# the table of step times
LAYOUTS = [((2, 0, 8), 1, (300, 150)), ((2, 0, 12), 1, (400, 250)), ((6, 0, 8), 1, (560, 700)),
           ((0, 2, 8), 2, (400, 251)), ((0, 4, 8), 2, (400, 400)), ((0, 4, 8), 2, (1001, 501)), ((0, 8, 8), 2, (900, 800)),
           ((2, 2, 8), 3, (200, 100)), ((6, 8, 8), 3, (300, 300))]


def test_all_layouts_are_named():
    """The table of layouts in the library has no other than those tested below."""
    import os
    import re
    src = open(os.path.join(os.path.dirname(__file__), "..", "taichirtm_b200", "csrc", "rtm_api.cu")).read()
    table = src[src.index("RES_LAYOUTS[] = {"):]
    rows = re.findall(r"\{RTM_\w+, (\d+), (\d+), (\d+), \{", table[: table.index("};")])
    assert {tuple(map(int, r)) for r in rows} == {k for k, _, _ in LAYOUTS} and len(rows) == 8


@pytest.mark.parametrize("layout,modes,grid", LAYOUTS)
@pytest.mark.parametrize("topography", [False, True])
def test_layout(layout, modes, grid, topography):
    from taichirtm_b200.plan import ShotGeometry
    nx, nz = grid
    surface = None
    if topography:
        surface = np.ones((nx, nz), np.float32)
        surface[: nx // 2, :2] = 0
        surface[nx // 2: nx // 2 + 9, 3] = 0.25
    src, rec = _points(nx, nz, dense=True)
    shots = [ShotGeometry(0, nx, src, rec)]
    assert _layout(nx, nz, modes, shots, surface)[:4] == layout + (1,)
    wav = _wavelets(len(src), 14)
    a = _run(shots, nx, nz, 14, 30, modes, None, wav, 5, 6, surface, resident=True)
    _same(a, _run(shots, nx, nz, 14, 30, modes, STREAM, wav, 5, 6, surface, resident=False))


@pytest.mark.parametrize("modes", [1, 3])
def test_batches_in_several_launches(modes):
    """Windowed P-SV shots, and shots of both wave types, more than a launch holds."""
    from taichirtm_b200.plan import ShotGeometry
    nx, nz, nt = 900, 330, 11
    shots = []
    for k in range(30):
        w = 220 + 37 * k % 200
        src, rec = _points(w, nz, dense=k % 3 == 0)
        shots.append(ShotGeometry((41 * k) % (nx - w), w, src, rec))
    assert _layout(nx, nz, modes, shots)[3] > 1
    wav = _wavelets(sum(len(s.src) for s in shots), nt)
    a = _run(shots, nx, nz, nt, 20, modes, None, wav, 4, 5, resident=True)
    _same(a, _run(shots, nx, nz, nt, 20, modes, STREAM, wav, 4, 5, resident=False))


def test_images_that_do_not_fit_beside_many_receivers():
    """600 receivers in one tile of two rows per lane: three such tiles fit on an SM,
    but not with their images, which stay in global memory then."""
    from taichirtm_b200.plan import ShotGeometry
    nx, nz, nt = 400, 350, 15
    src, rec = _points(nx, nz, dense=False)
    block = np.array([[200 + i, 112 + j] for i in range(12) for j in range(50)], np.int32)
    shots = [ShotGeometry(0, nx, src, np.concatenate([rec, block]))]
    assert _layout(nx, nz, 1, shots) == (2, 0, 8, 1, 0)
    wav = _wavelets(len(src), nt)
    a = _run(shots, nx, nz, nt, 20, 1, None, wav, 1, 4, resident=True)
    _same(a, _run(shots, nx, nz, nt, 20, 1, STREAM, wav, 1, 4, resident=False))


@pytest.mark.parametrize("store", ["f32", "f16", "bf16", "i16"])
@pytest.mark.parametrize("every,check", [(5, 4), (8, 1), (6, 3), (23, 5)])
def test_shot_that_fails_under_checkpoints(store, every, check):
    """One of two shots overflows at step 9 of the forward pass, and the backward
    pass of data that overflow it, too: status codes, seismograms, checkpoints and
    images are the streaming kernels'; the other shot goes on."""
    from taichirtm_b200 import _lib
    from taichirtm_b200.plan import Plan, ShotGeometry, _i32p, _ptr, _stream, check as ok
    nx, nz, nt, fw = 230, 131, 23, 12
    shots = [ShotGeometry(0, 121, *_points(121, nz, dense=True)), ShotGeometry(99, 131, *_points(131, nz, dense=True))]
    wav = _wavelets(sum(len(s.src) for s in shots), nt)
    wav[:, 0, 9] = 3e38
    wav = torch.as_tensor(wav).cuda()
    obs0 = torch.as_tensor(_wavelets(sum(len(s.rec) for s in shots), nt, 5)).cuda()
    obs0[:, 3, nt - 1 - 10] = 3e38  # reached at loop step 10
    L, dt, res = _lib.lib(), _lib.CKPT_DTYPES[store], []
    for tune in (None, dict(vec=2, rows=9, warps=2, tsteps=1)):
        p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, fw, 1, shots, tune=tune)
        p.set_model(*_model(nx, nz))
        assert p.resident() == (tune is None)
        ck = torch.zeros(max(int(L.rtm_plan_checkpoint_bytes(p.h, every, dt)), 1), dtype=torch.uint8, device="cuda")
        seis = torch.zeros((3, p.nrec_total, nt), device="cuda")
        stack = torch.zeros((3, nx, nz), dtype=torch.float64, device="cuda")
        flags, flags_b = np.zeros(2, np.int32), np.zeros(2, np.int32)
        ok(L.rtm_forward_checkpointed(p.h, _ptr(wav), _ptr(seis), every, dt, _ptr(ck), check, _i32p(flags), _stream()), "f")
        calm = wav.clone()
        calm[:, 0, 9] = 0.0
        ck2 = torch.zeros_like(ck)
        seis2 = torch.zeros_like(seis)
        f2 = np.zeros(2, np.int32)
        ok(L.rtm_forward_checkpointed(p.h, _ptr(calm), _ptr(seis2), every, dt, _ptr(ck2), check, _i32p(f2), _stream()), "f")
        ok(L.rtm_backward_checkpointed(p.h, _ptr(calm), _ptr(obs0), every, dt, _ptr(ck2), 2, None, _ptr(stack), check,
                                       _i32p(flags_b), _stream()), "b")
        assert flags[0] > 0 and flags[1] == 0 and f2.max() == 0 and flags_b[0] > 0 and flags_b[1] == 0
        # the padding of FP32 slots is not compared (it is not read)
        res.append([flags, flags_b] + [x.cpu().numpy() for x in (seis, seis2, stack)] + ([ck.cpu().numpy(), ck2.cpu().numpy()] if dt else []))
        p.close()
    assert np.count_nonzero(res[0][4][:, 160:]) > 0  # rows of the second shot alone
    _same(*res)
