"""Launch shapes and the states of a plan that callers can reach: every accepted
shape runs, with the results of the one-step kernel (tolerance 0), whichever
form of a kernel and whichever path the library takes for it."""
import numpy as np
import pytest
import torch

from tests.test_gpu_resident import _model, _points, _run, _same, _wavelets

pytestmark = pytest.mark.gpu
STREAM = dict(vec=2, rows=5, warps=2, tsteps=1)


def _topography(nx, nz):
    surface = np.ones((nx, nz), np.float32)
    surface[: nx // 2, :2] = 0
    return surface


@pytest.mark.parametrize("modes", [1, 2, 3])
@pytest.mark.parametrize("vec", [2, 4])
@pytest.mark.parametrize("warps", [7, 8])
def test_widest_ring_shapes_run_with_a_mask(modes, vec, warps):
    """The rings of 8 warps with 4 columns per lane, both wave types and a mask
    exceed a CTA's shared memory: the state stays in registers then."""
    from taichirtm_b200.plan import ShotGeometry
    nx, nz, nt = 70, 130, 8  # no single steps: their kernel has no room for 8 such warps either
    src, rec = _points(nx, nz, dense=True)
    shots = [ShotGeometry(0, nx, src, rec)]
    wav, mask = _wavelets(len(src), nt), _topography(nx, nz)
    tune = dict(vec=vec, rows=6, warps=warps, prefetch=3, tsteps=2)
    a = _run(shots, nx, nz, nt, 12, modes, tune, wav, 2, 0, mask, resident=False)
    _same(a, _run(shots, nx, nz, nt, 12, modes, STREAM, wav, 2, 0, mask, resident=False))


@pytest.mark.parametrize("vec,prefetch,warps", [(2, 3, 2), (2, 4, 1), (4, 3, 4), (4, 4, 1), (2, 1, 4), (2, 1, 8), (4, 1, 4)])
@pytest.mark.parametrize("modes,mask", [(1, False), (1, True), (2, False), (3, False), (3, True)])
def test_shapes_with_many_tasks(modes, mask, vec, prefetch, warps):
    """Launches of 12 tasks per SM and more may bring the state through a ring, or
    use packed arithmetic; the tests on small grids run the other forms."""
    from taichirtm_b200.plan import ShotGeometry
    nx, nz, nt = 810, 370, 7
    src, rec = _points(nx, nz, dense=True)
    shots = [ShotGeometry(0, nx, src, rec)]
    wav, surface = _wavelets(len(src), nt), _topography(nx, nz) if mask else None
    tune = dict(vec=vec, rows=1, warps=warps, prefetch=prefetch, tsteps=2)
    a = _run(shots, nx, nz, nt, 12, modes, tune, wav, 2, 4, surface, resident=False)
    _same(a, _run(shots, nx, nz, nt, 12, modes, STREAM, wav, 2, 4, surface, resident=False))


@pytest.mark.parametrize("vec,prefetch", [(2, 1), (2, 3), (4, 3)])
@pytest.mark.parametrize("store", ["f32", "i16"])
def test_checkpoints_and_recompute_with_many_tasks(store, vec, prefetch):
    """The storing forms of the same launches: checkpoints, the states that the
    adjoint recomputes, and what is made of them."""
    import ctypes
    from taichirtm_b200 import _lib
    from taichirtm_b200.plan import Plan, ShotGeometry, _i32p, _ptr, _stream, check as ok
    nx, nz, nt, every = 810, 370, 11, 5
    src, rec = _points(nx, nz, dense=False)
    shots = [ShotGeometry(0, nx, src, rec)]
    wav = torch.as_tensor(_wavelets(len(src), nt)).cuda()
    L, dt, res = _lib.lib(), _lib.CKPT_DTYPES[store], []
    for tune in (dict(vec=vec, rows=1, warps=2, tsteps=2, prefetch=prefetch), dict(STREAM, vec=vec)):
        p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 12, 1, shots, tune=tune)
        p.set_model(*_model(nx, nz))
        ck = torch.zeros(int(L.rtm_plan_checkpoint_bytes(p.h, every, dt)), dtype=torch.uint8, device="cuda")
        seis = torch.zeros((3, p.nrec_total, nt), device="cuda")
        stack = torch.zeros((3, nx, nz), dtype=torch.float64, device="cuda")
        grad = torch.zeros((5, nx, nz), dtype=torch.float64, device="cuda")
        flags = np.zeros(1, np.int32)
        ok(L.rtm_forward_checkpointed(p.h, _ptr(wav), _ptr(seis), every, dt, _ptr(ck), 4, _i32p(flags), _stream()), "f")
        ok(L.rtm_backward_checkpointed(p.h, _ptr(wav), _ptr(seis), every, dt, _ptr(ck), 2, None, _ptr(stack), 4, _i32p(flags),
                                       _stream()), "b")
        ok(L.rtm_adjoint(p.h, _ptr(wav), _ptr(seis), every, dt, _ptr(ck), _ptr(grad), ctypes.c_void_p(0), _stream()), "a")
        res.append([x.cpu().numpy() for x in (seis, ck, stack, grad)])
        p.close()
    assert np.abs(res[0][2]).max() > 0 and np.abs(res[0][3]).max() > 0
    _same(*res)


def test_prefetch_zero_is_a_launch_shape():
    """prefetch 0 by itself asks for plain row loads, so the plan streams; a negative
    one, like no launch shape at all, leaves the choice to the library."""
    from taichirtm_b200.plan import ShotGeometry
    nx, nz, nt = 40, 30, 6
    src, rec = _points(nx, nz, dense=False)
    shots = [ShotGeometry(0, nx, src, rec)]
    wav = _wavelets(len(src), nt)
    a = _run(shots, nx, nz, nt, 4, 3, dict(prefetch=0), wav, 2, 0, resident=False)
    _same(a, _run(shots, nx, nz, nt, 4, 3, dict(prefetch=-1, graphs=1), wav, 2, 0, resident=True))


@pytest.mark.parametrize("tune", [None, dict(vec=2, rows=5, warps=2, tsteps=1), dict(vec=2, rows=5, warps=2, tsteps=2),
                                  dict(vec=4, rows=5, warps=1, tsteps=2, prefetch=4, graphs=1)])
@pytest.mark.parametrize("nt,check", [(12, 1), (13, 3), (14, 5), (14, 3)])
def test_wavefield_of_a_stopped_shot(tune, nt, check):
    """The wavefield of a shot that stopped is the one of its last step, the step
    whose check failed, however the plan runs; other shots go on to the end."""
    from taichirtm_b200.plan import Plan, ShotGeometry
    nx, nz, w, fw, at = 90, 40, 50, 5, 3
    rec = np.array([[i, 1] for i in range(w)], np.int32)
    shots = [ShotGeometry(0, w, np.array([[25, 20]], np.int32), rec), ShotGeometry(40, w, np.array([[25, 20]], np.int32), rec)]
    # dt dx dz / rho of it, 1e33, is above the check's limit of 1e30 at step `at`
    wav = _wavelets(2, nt)
    wav[:, 0, at] = 3e38
    last = -(-at // check) * check
    mu, lam, rho = _model(nx, nz)
    p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, fw, 1, shots, tune=tune)
    p.set_model(mu, lam, rho)
    flags, _, _, _ = p.forward(torch.as_tensor(wav), check_interval=check)
    assert flags[0] > 0 and flags[1] == 0
    got = [p.wavefield(k).cpu().numpy() for k in range(2)]
    p.close()
    # the same shots by themselves, over the steps each ran, without checks
    for k, steps in ((0, last + 1), (1, nt)):
        q = Plan(nx, nz, 4.0, 4.0, steps, 2000.0, fw, 1, [shots[k]], tune=STREAM)
        q.set_model(mu, lam, rho)
        q.forward(torch.as_tensor(np.ascontiguousarray(wav[:, k:k + 1, :steps])), check_interval=0)
        assert np.array_equal(got[k], q.wavefield(0).cpu().numpy(), equal_nan=True)
        q.close()


@pytest.mark.parametrize("modes", [1, 3])
@pytest.mark.parametrize("tune", [dict(vec=2, rows=9, warps=2, tsteps=2, graphs=1), dict(vec=2, rows=9, warps=2, tsteps=2, prefetch=3, graphs=1),
                                  dict(vec=4, rows=9, warps=2, tsteps=1, graphs=1), None])
def test_mask_added_and_dropped_on_one_plan(tune, modes):
    """set_model decides whether there is a mask, also after loops that were
    captured or laid out for the other case."""
    from taichirtm_b200.plan import Plan, ShotGeometry
    nx, nz, nt = 90, 75, 11
    src, rec = _points(nx, nz, dense=True)
    shots = [ShotGeometry(0, nx, src, rec)]
    wav = torch.as_tensor(_wavelets(len(src), nt)).cuda()
    model, mask = _model(nx, nz), _topography(nx, nz)

    def passes(p, snaps=None):
        out = []
        f, seis, snaps, isn = p.forward(wav, save=True, isnap=2, check_interval=0, snaps=snaps)
        _, img, _ = p.backward(seis, snaps, isn, len(isn), 2, check_interval=0)
        return [seis.cpu().numpy(), img.cpu().numpy()], snaps

    want = {}
    for has in (False, True):
        q = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 8, modes, shots, tune=STREAM)
        q.set_model(*model, mask if has else None)
        want[has], _ = passes(q)
        q.close()
    assert not np.array_equal(want[False][0], want[True][0])
    p, snaps = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 8, modes, shots, tune=tune), None
    for has in (False, True, False, True, True, False):
        p.set_model(*model, mask if has else None)
        got, snaps = passes(p, snaps)
        _same(got, want[has])
    assert p.resident() == (tune is None)
    p.close()



@pytest.mark.parametrize("tune", [dict(vec=2, rows=9, warps=2, tsteps=2), dict(vec=4, rows=9, warps=2, tsteps=1, prefetch=3)])
def test_graph_replays_of_streaming_plans(tune):
    """Time loops captured once and replayed give what direct launches give: on the
    capturing call, on replays with other data in the same buffers, and after the
    snapshot schedule has changed and changed back."""
    from taichirtm_b200.plan import Plan, ShotGeometry
    nx, nz, nt = 90, 75, 17
    src, rec = _points(nx, nz, dense=True)
    res = []
    for graphs in (0, 1):
        p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 8, 3, [ShotGeometry(0, nx, src, rec)], tune=dict(tune, graphs=graphs))
        p.set_model(*_model(nx, nz))
        assert not p.resident()
        wav = torch.empty((3, len(src), nt), device="cuda")
        bufs, out = {i: [p.snapshot_buffer(nt // i) for _ in range(3)] for i in (2, 3)}, []
        for seed, isnap in ((1, 2), (2, 2), (3, 3), (4, 3), (5, 2)):
            wav.copy_(torch.as_tensor(_wavelets(len(src), nt, seed)))
            f, seis, snaps, isn = p.forward(wav, save=True, isnap=isnap, check_interval=4, snaps=bufs[isnap])
            fb, img, _ = p.backward(seis, snaps, isn, len(isn), isnap, check_interval=4)
            out += [f, fb, seis.cpu().numpy(), img.cpu().numpy()] + [p.snapshot_view(b, len(isn)).cpu().numpy() for b in snaps]
        res.append(out)
        p.close()
    assert np.abs(res[0][2]).max() > 0 and np.abs(res[0][3]).max() > 0
    _same(*res)



def test_captured_calls_outlive_a_change_of_the_mask():
    """A forward call that a caller captured (flags NULL) replays after set_model has
    added a mask, with the buffers and the maskless loop it was captured with.  A
    set_model that meets a mask for the first time can be captured, too."""
    from taichirtm_b200 import _lib
    from taichirtm_b200._lib import check as ok
    from taichirtm_b200.plan import Plan, ShotGeometry, _ptr, _stream
    nx, nz, nt = 300, 150, 21
    src, rec = _points(nx, nz, dense=False)
    shots, L = [ShotGeometry(0, nx, src, rec)], _lib.lib()
    model = [torch.as_tensor(x).cuda() for x in _model(nx, nz)]
    mask, wav = torch.as_tensor(_topography(nx, nz)).cuda(), torch.as_tensor(_wavelets(len(src), nt)).cuda()
    want = {}
    for has in (False, True):
        q = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 20, 3, shots, tune=STREAM)
        q.set_model(*model, mask if has else None)
        want[has] = q.forward(wav)[1]
        q.close()
    assert not torch.equal(want[False], want[True])
    p, seis, none = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 20, 3, shots), torch.zeros_like(want[False]), None

    def call():
        ok(L.rtm_forward(p.h, _ptr(wav), _ptr(seis), 0, 1, none, none, none, none, 0, none, _stream()), "rtm_forward")

    def replay(graph):
        seis.zero_()
        graph.replay()
        ok(L.rtm_plan_status(p.h, none, _stream()), "rtm_plan_status")
        return seis
    p.set_model(*model)
    assert p.resident() and torch.equal(p.forward(wav)[1], want[False])
    plain, masked = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(plain):
        call()
    assert torch.equal(replay(plain), want[False])
    with torch.cuda.graph(masked):
        p.set_model(*model, mask)
        call()
    assert not p.resident() and torch.equal(replay(masked), want[True])
    p.set_model(*model, mask)
    assert p.resident() and torch.equal(p.forward(wav)[1], want[True])
    assert torch.equal(replay(plain), want[False]) and torch.equal(replay(masked), want[True])
    p.set_model(*model)
    assert p.resident() and torch.equal(p.forward(wav)[1], want[False])
    del plain, masked
    p.close()


def test_plan_streams_when_its_resident_buffers_do_not_fit():
    """A plan whose own buffers fit in the device memory that is left, but not
    those of the resident loops too, is made all the same and streams."""
    from taichirtm_b200.plan import Plan, ShotGeometry
    nx, nz, nt = 560, 700, 6
    src, rec = _points(nx, nz, dense=False)
    shots = [ShotGeometry(0, nx, src, rec)]
    wav, model = torch.as_tensor(_wavelets(len(src), nt)).cuda(), [torch.as_tensor(x).cuda() for x in _model(nx, nz)]

    def make(tune):
        p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 20, 1, shots, tune=tune)
        p.set_model(*model)
        return p

    def used(tune):  # device memory that a plan of this shape takes
        before = torch.cuda.mem_get_info()[0]
        p = make(tune)
        n, resident = before - torch.cuda.mem_get_info()[0], p.resident()
        seis = p.forward(wav)[1]
        p.close()
        return n, resident, seis

    used(None)  # one-time loading of the kernels
    (n_stream, r_stream, want), (n_res, r_res, seis) = used(STREAM), used(None)
    assert r_res and not r_stream and torch.equal(want, seis) and n_res - n_stream > 16 << 20
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (n_stream + n_res) // 2, dtype=torch.uint8, device="cuda")
    p = make(None)
    resident = p.resident()
    del hold
    torch.cuda.empty_cache()
    assert not resident and torch.equal(p.forward(wav)[1], want)
    p.close()


WAIT = r'''
import numpy as np, torch
from taichirtm_b200 import _lib
from taichirtm_b200._lib import RtmError, check as ok
from taichirtm_b200.plan import Plan, ShotGeometry, _i32p, _ptr, _stream
from tests.test_gpu_resident import _model, _points, _wavelets
nx, nz, nt = 300, 150, 40
src, rec = _points(nx, nz, dense=False)
p = Plan(nx, nz, 4.0, 4.0, nt, 2000.0, 20, 1, [ShotGeometry(0, nx, src, rec)])
p.set_model(*_model(nx, nz))
assert p.resident()
L, wav = _lib.lib(), torch.as_tensor(_wavelets(len(src), nt)).cuda()
want = p.forward(wav)[1].clone()
seis, flags, none = torch.zeros_like(want), np.zeros(1, np.int32), None

def forward(flags):
    return L.rtm_forward(p.h, _ptr(wav), _ptr(seis), 0, 1, none, none, none, none, 0, flags, _stream())

def status():
    return L.rtm_plan_status(p.h, _i32p(flags), _stream())

assert forward(none) == 0 and status() == 0 and torch.equal(seis, want)
ok(L.rtm_plan_set_wait_limit(p.h, 1), "limit")
forward(none)
assert status() == -2 and b"ran out" in L.rtm_last_error()
assert status() == 0  # reported once
assert forward(_i32p(flags)) == -2 and status() == 0
try:
    p.backward(want, None, [], 0, 1)
    raise SystemExit("backward reported nothing")
except RtmError:
    pass
forward(none)
ok(L.rtm_plan_set_wait_limit(p.h, 0), "limit")
forward(none)  # complete itself, and does not hide the one before
assert status() == -2 and torch.equal(seis, want)
assert forward(_i32p(flags)) == 0 and torch.equal(seis, want)
print("WAIT_OK")
'''


def test_wait_that_runs_out_is_reported():
    """A wait limit of one poll (bounds-checking build): no packet of a neighbouring
    tile is there by then, so the tiles leave at their first exchange and the
    results are incomplete.  Calls with flags say so; the others leave it to the
    next report."""
    from tests.test_gpu_bounds import _child
    r = _child(WAIT, timeout=300)
    assert r.returncode == 0 and "WAIT_OK" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
