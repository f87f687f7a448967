"""GPU: what one call of a context leaves for the next.

A context keeps its buffers between calls.  Passes that follow a slab run, a refused call or a failed
allocation give what a fresh context gives; they run the same kernels on the same values, so the
results are equal bit for bit.
"""
import contextlib

import numpy as np
import pytest
import torch

from cases import random_signals
from elasticisolib_3d_b200 import _native as N
from elasticisolib_3d_b200 import synthetic as S
from elasticisolib_3d_b200.engine import Propagator, SlabPropagator, _geom, checkpoint_plan
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DTW = 0.0005


def _medium(nz, nx, ny):
    el = S.elastic_from_velocity(*S.gaussian_perturbed_model((ny, nx, nz), 2500.0, 1443.0, 2000.0, 0.1, 2.0, 5))
    return O.medium_planes(el, DTW, np.float32)


def _points(rng, nz, nx, ny, n):
    z, x, y = (rng.integers(4, m - 4, size=4 * n) for m in (nz, nx, ny))
    return np.unique((y * nx + x) * nz + z)[:n].astype(np.int64)


def _propagator(nz, nx, ny, nts, sub=4, pad=3, cls=Propagator, **kw):
    return cls(nz, nx, ny, nts, sub, pad, 10.0, 10.0, 10.0, sub * DTW, **kw)


def _equal(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@contextlib.contextmanager
def _memory_left(nbytes):
    """All but about `nbytes` of the device's free memory held by another allocation."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - int(nbytes), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        torch.cuda.synchronize()
        del hog
        torch.cuda.empty_cache()


def _device_sets(rng, nz, nx, ny, nts, nsrc=5, nrec=200):
    """Explosive sources and pressure-like receivers as device tables, and random source signals."""
    s = _points(rng, nz, nx, ny, nsrc)
    r = np.unique(np.concatenate([s, _points(rng, nz, nx, ny, nrec)]))
    so = [len(s) * min(max(k - 3, 0), 3) for k in range(10)]
    ro = [len(r) * min(max(k - 3, 0), 3) for k in range(10)]
    sig = torch.from_numpy(rng.standard_normal((nts, so[9])).astype(np.float32)).cuda()
    return torch.from_numpy(np.tile(s, 3)).cuda(), so, torch.from_numpy(np.tile(r, 3)).cuda(), ro, sig


@pytest.mark.parametrize("first", [False, True])
def test_born_image_after_a_slab_run(first):
    """A slab run leaves its neighbours' planes in the ghost planes of the working levels, which the
    imaging pass's ring of levels takes over (first: the ring exists before the slab run)."""
    nz, nx, ny, nts = 40, 33, 50, 12
    rng = np.random.default_rng(1)
    med = _medium(nz, nx, ny)
    spos = [_points(rng, nz, nx, ny, 4) for _ in range(7)]
    rpos = [_points(rng, nz, nx, ny, 60) for _ in range(7)]
    sl = _propagator(nz, nx, ny, nts, cls=SlabPropagator, devices=(0, 0))
    sl.set_medium(med)
    part, ny0 = sl.slabs[0], sl.sizes[0]
    lspos = [_points(rng, nz, nx, ny0, 4) for _ in range(7)]
    lrpos = [_points(rng, nz, nx, ny0, 60) for _ in range(7)]
    sig, dat = random_signals(lspos, nts, rng), random_signals(lrpos, nts, rng)
    if first:
        part.born_adjoint(sig, dat, lspos, lrpos)
    sl.nl_forward([1e3 * s for s in random_signals(spos, nts, rng)], spos, rpos)
    got = part.born_adjoint(sig, dat, lspos, lrpos)
    fresh = _propagator(nz, nx, ny0, nts)
    fresh.set_medium(med[:, :ny0])
    _equal(got, fresh.born_adjoint(sig, dat, lspos, lrpos))
    fresh.close()
    sl.close()


def test_born_calls_refuse_a_missing_plane():
    """A null perturbation or image plane is refused with a status, on planes large enough for the
    staged copies too, and the next call runs."""
    nz, nx, ny, nts = 168, 168, 152, 3
    rng = np.random.default_rng(6)
    pr = _propagator(nz, nx, ny, nts, sub=1)
    pr.set_medium(_medium(nz, nx, ny))
    spos = [_points(rng, nz, nx, ny, 4) for _ in range(7)]
    rpos = [_points(rng, nz, nx, ny, 9) for _ in range(7)]
    sig, dat = random_signals(spos, nts, rng), random_signals(rpos, nts, rng)
    pert = [np.ones((ny, nx, nz), np.float32)] * 8
    SP, SN, k1 = _geom(spos)
    RP, RN, k2 = _geom(rpos)
    ref = pr.born_forward(sig, pert, spos, rpos)
    for hole in (0, 7):
        planes = [None if k == hole else p for k, p in enumerate(pert)]
        for name in ("e3d_born_forward", "e3d_born_adjoint"):
            with pytest.raises(N.E3DError, match="null"):
                N.call(name, pr.handle, N.ptr_array(sig), N.ptr_array(dat), SP, SN, RP, RN, N.ptr_array(planes))
    _equal(pr.born_forward(sig, pert, spos, rpos), ref)
    pr.close()


def test_failed_allocation_leaves_the_medium():
    """A call that runs out of memory, whatever it gave up on the way, leaves a medium that the next
    call propagates in."""
    nz, nx, ny, nts = 72, 400, 800, 4
    rng = np.random.default_rng(2)
    med = _medium(nz, nx, ny)
    sp, so, rp, ro, sig = _device_sets(rng, nz, nx, ny, nts)
    out = []
    for short in (False, True):
        pr = _propagator(nz, nx, ny, nts)
        pr.set_medium(med)
        rec = torch.empty((nts, ro[9]), device="cuda")
        with pytest.raises(N.E3DError):  # refused; the position check has its word of memory from here on
            pr.nl_propagate_device(False, torch.zeros_like(sp), so, rp, ro, sig, rec)
        pr.synchronize()
        if short:
            with _memory_left(8 << 20):
                with pytest.raises(N.E3DError):
                    pr.nl_propagate_device(False, sp, so, rp, ro, sig, rec)
        pr.nl_propagate_device(False, sp, so, rp, ro, sig, rec)
        pr.synchronize()
        out.append(rec.cpu().numpy())
        pr.close()
    assert np.abs(out[0]).max() > 0
    np.testing.assert_array_equal(out[1], out[0])


def test_refused_plan_keeps_the_buffers():
    """A budget that no plan fits is refused without giving up what the context holds: a propagation
    before and after it uses the same memory."""
    nz, nx, ny, nts = 72, 200, 400, 4
    rng = np.random.default_rng(7)
    pr = _propagator(nz, nx, ny, nts)
    pr.set_medium(_medium(nz, nx, ny))
    sp, so, rp, ro, sig = _device_sets(rng, nz, nx, ny, nts)
    rec = torch.empty((nts, ro[9]), device="cuda")
    pr.nl_propagate_device(False, sp, so, rp, ro, sig, rec)
    pr.set_checkpoint_policy("auto", 0, 1.0)
    with pytest.raises(N.E3DError):
        pr.fwi_forward_device(sp, so, rp, ro, sig, rec)
    pr.synchronize()
    before = torch.cuda.mem_get_info()[0]
    pr.nl_propagate_device(False, sp, so, rp, ro, sig, rec)
    pr.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 4 * nz * nx * ny
    pr.close()


@pytest.mark.parametrize("nz,nx,ny,nts,budget", [(104, 104, 96, 300, 4.0e9), (72, 100, 100, 400, 3.6e9),
                                                 (65, 70, 80, 200, 0.95e9), (104, 104, 96, 300, 2.0e9),
                                                 (104, 104, 96, 300, 1.0e9)])
def test_rows_do_not_change_the_memory_plan(nz, nx, ny, nts, budget):
    """The plan of the checkpointed passes is the one of the grid's own cells (checkpoint_plan),
    however the context lays out its rows."""
    rng = np.random.default_rng(4)
    pr = _propagator(nz, nx, ny, nts)
    pr.set_medium(_medium(nz, nx, ny))
    pr.set_checkpoint_policy("auto", 0, budget)
    sp, so, rp, ro, sig = _device_sets(rng, nz, nx, ny, nts)
    pr.fwi_forward_device(sp, so, rp, ro, sig, torch.empty((nts, ro[9]), device="cuda"))
    pr.synchronize()
    want = checkpoint_plan(nz * nx * ny, ny, nts, budget)
    assert (pr.checkpoint_type, pr.velocity_storage, pr.checkpoint_segment) == want[:3]
    pr.close()


def test_staged_planes_in_and_out():
    """Image planes of 17 MB sent and fetched through the staging buffers: zero data leaves the caller's
    planes as they were."""
    nz, nx, ny, nts = 168, 168, 152, 3
    rng = np.random.default_rng(8)
    pr = _propagator(nz, nx, ny, nts, sub=1)
    pr.set_medium(_medium(nz, nx, ny))
    spos = [_points(rng, nz, nx, ny, 4) for _ in range(7)]
    rpos = [_points(rng, nz, nx, ny, 9) for _ in range(7)]
    sig, dat = random_signals(spos, nts, rng), [0 * d for d in random_signals(rpos, nts, rng)]
    for _ in range(2):
        init = [rng.standard_normal((ny, nx, nz), dtype=np.float32) for _ in range(8)]
        _equal(pr.born_adjoint(sig, dat, spos, rpos, init), init)
    pr.close()


@pytest.mark.parametrize("nz,nx,ny", [(16, 9, 10), (17, 13, 11), (72, 40, 20), (101, 30, 21), (168, 200, 188)])
def test_medium_from_host_and_device(nz, nx, ny):
    """The medium from host planes, from device planes and from device planes off the 16-byte grid gives
    the same traces (rows below and above a warp, of every remainder mod 4, one part and several)."""
    nts = 4
    rng = np.random.default_rng(9)
    med = _medium(nz, nx, ny)
    sp, so, rp, ro, sig = _device_sets(rng, nz, nx, ny, nts)
    flat = torch.empty(med.size + 1, device="cuda")
    off = flat[1:].view(med.shape)
    off.copy_(torch.from_numpy(med))
    out = []
    for m in (med, torch.from_numpy(med).cuda(), off):
        torch.cuda.synchronize()
        pr = _propagator(nz, nx, ny, nts)
        pr.set_medium(m)
        rec = torch.empty((nts, ro[9]), device="cuda")
        pr.nl_propagate_device(False, sp, so, rp, ro, sig, rec)
        pr.synchronize()
        out.append(rec.cpu().numpy())
        pr.close()
    assert np.abs(out[0]).max() > 0
    _equal(out[1:], [out[0]] * 2)


def test_first_medium_fits_without_padding():
    """Memory for the medium's planes in unpadded rows only (72-cell rows: a third more when padded)."""
    nz, nx, ny, nts = 72, 200, 400, 4
    rng = np.random.default_rng(10)
    med = _medium(nz, nx, ny)
    sp, so, rp, ro, sig = _device_sets(rng, nz, nx, ny, nts)
    out = []
    for short in (False, True):
        pr = _propagator(nz, nx, ny, nts)
        with _memory_left(9.5 * 4 * nz * nx * ny) if short else contextlib.nullcontext():
            pr.set_medium(med)
        rec = torch.empty((nts, ro[9]), device="cuda")
        pr.nl_propagate_device(False, sp, so, rp, ro, sig, rec)
        pr.synchronize()
        out.append(rec.cpu().numpy())
        pr.close()
    np.testing.assert_array_equal(out[1], out[0])


def _gradient(pr, sets, nts, ny, nx, nz, short=None):
    """Predicted traces and gradient planes of the traces themselves; short: memory left for the
    gradient pass."""
    sp, so, rp, ro, sig = sets
    rec = torch.empty((nts, ro[9]), device="cuda")
    grad = torch.zeros((8, ny, nx, nz), device="cuda")
    pr.fwi_forward_device(sp, so, rp, ro, sig, rec)
    pr.synchronize()
    with _memory_left(short) if short else contextlib.nullcontext():
        pr.fwi_gradient_device(sp, so, rp, ro, sig, rec, grad)
        pr.synchronize()
    return rec.cpu().numpy(), grad.cpu().numpy()


def test_gradient_after_a_forward_that_ran_out_of_memory():
    """A checkpointed forward that found no memory for all its levels leaves what it got to the next,
    which runs once there is more."""
    nz, nx, ny, nts = 72, 200, 400, 6
    rng = np.random.default_rng(11)
    med = _medium(nz, nx, ny)
    sets = _device_sets(rng, nz, nx, ny, nts)
    out = []
    for short in (False, True):
        pr = _propagator(nz, nx, ny, nts)
        pr.set_medium(med)
        pr.set_checkpoint_policy("fp32", 2)
        pr.set_velocity_storage("fp32")
        if short:
            sp, so, rp, ro, sig = sets
            rec = torch.empty((nts, ro[9]), device="cuda")
            pr.synchronize()
            with _memory_left(24 * 4 * nz * nx * ny):
                with pytest.raises(N.E3DError, match="memory"):
                    pr.fwi_forward_device(sp, so, rp, ro, sig, rec)
                torch.cuda.synchronize()
                held = torch.cuda.mem_get_info()[0]
                with pytest.raises(N.E3DError, match="memory"):
                    pr.fwi_forward_device(sp, so, rp, ro, sig, rec)
                torch.cuda.synchronize()
                assert torch.cuda.mem_get_info()[0] >= held
        out.append(_gradient(pr, sets, nts, ny, nx, nz))
        pr.close()
    _equal(out[1], out[0])


def test_gradient_fits_without_padding():
    """A gradient whose forward had room for padded rows and which has room for its own fields in
    unpadded ones only (72-cell rows: a third more when padded): the planes of one with the room."""
    nz, nx, ny, nts, sub = 72, 200, 400, 6, 4
    rng = np.random.default_rng(12)
    med = _medium(nz, nx, ny)
    sets = _device_sets(rng, nz, nx, ny, nts)
    out = []
    for short in (None, 1.15 * (sub + 2) * 9 * 4 * nz * nx * ny):  # the adjoint ring and a carried block
        pr = _propagator(nz, nx, ny, nts, sub)
        pr.set_medium(med)
        pr.set_checkpoint_policy("fp32", 2)
        pr.set_velocity_storage("fp32")
        out.append(_gradient(pr, sets, nts, ny, nx, nz, short))
        pr.close()
    assert np.abs(out[0][1]).max() > 0
    _equal(out[1], out[0])


@pytest.mark.parametrize("what", ["slabs", "steps"])
def test_levels_fit_without_padding(what):
    """Slab runs and bare steps with room for their two levels in unpadded rows only (72-cell rows: a
    third more when padded)."""
    nz, nx, ny, nts = 72, 200, 400, 4
    rng = np.random.default_rng(13)
    med = _medium(nz, nx, ny)
    left = 1.15 * 18 * 4 * nz * nx * ny
    if what == "steps":
        pr = _propagator(nz, nx, ny, nts)
        pr.set_medium(med)
        pr.synchronize()
        with _memory_left(left):
            pr.step_only(0, 2)
            pr.synchronize()
        pr.close()
        return
    spos = [_points(rng, nz, nx, ny, 4) for _ in range(7)]
    rpos = [np.unique(np.concatenate([p, _points(rng, nz, nx, ny, 60)])) for p in spos]
    model = random_signals(spos, nts, rng)
    out = []
    for short in (False, True):
        sl = _propagator(nz, nx, ny, nts, cls=SlabPropagator, devices=(0, 0))
        sl.set_medium(med)
        torch.cuda.synchronize()
        with _memory_left(left) if short else contextlib.nullcontext():
            out.append(sl.nl_forward(model, spos, rpos))
        sl.close()
    assert max(np.abs(x).max() for x in out[0]) > 0
    _equal(out[1], out[0])


def test_admitted_shots_leave_the_rows():
    """Shots dealt into batches by the free memory fit in the rows the context has."""
    nz, nx, ny, nts, shots = 72, 200, 200, 3, 10
    rng = np.random.default_rng(14)
    spos = [[_points(rng, nz, nx, ny, 4) for _ in range(7)] for _ in range(shots)]
    rpos = [_points(rng, nz, nx, ny, 50) for _ in range(7)]
    models = [random_signals(sp, nts, rng) for sp in spos]
    pr = _propagator(nz, nx, ny, nts, q2compat=0)
    pr.set_medium(_medium(nz, nx, ny))
    cells = pr.field_cells
    assert cells == 96 * nx * ny
    whole = pr.nl_forward_batch(models, spos, rpos)
    pr.close()
    pr = _propagator(nz, nx, ny, nts, q2compat=0)
    pr.set_medium(_medium(nz, nx, ny))
    pr.synchronize()
    with _memory_left(1.1 * shots * 18 * 4 * nz * nx * ny + (64 << 20)):
        dealt = pr.nl_forward_shots(models, spos, rpos)
    assert pr.field_cells == cells
    for a, b in zip(dealt, whole):
        _equal(a, b)
    pr.close()


@pytest.mark.parametrize("surface", [0, 1])
@pytest.mark.parametrize("adjoint", [False, True])
def test_slabs_of_unlike_rows_equal_the_whole_grid(adjoint, surface):
    """Slabs of one grid, the first of which gave up its rows' padding: the traces of the undivided
    grid, with the free surface (applied in the stepper) too."""
    nz, nx, ny, nts = 72, 120, 300, 5
    rng = np.random.default_rng(15)
    med = _medium(nz, nx, ny)
    spos = [_points(rng, nz, nx, ny, 20) for _ in range(7)]
    rpos = [np.unique(np.concatenate([p, _points(rng, nz, nx, ny, 400)])) for p in spos]
    whole = _propagator(nz, nx, ny, nts, free_surface=surface)
    whole.set_medium(med)
    sl = _propagator(nz, nx, ny, nts, cls=SlabPropagator, devices=(0, 0), free_surface=surface)
    sl.set_medium(med)
    first, n0 = sl.slabs[0], nz * nx * sl.sizes[0]
    first.synchronize()
    with _memory_left(1.15 * 18 * 4 * n0):
        first.step_only(0, 1)
        first.synchronize()
    assert first.field_cells == n0 and sl.slabs[1].field_cells > nz * nx * sl.sizes[1]
    if adjoint:
        dat = random_signals(rpos, nts, rng)
        got, ref = sl.nl_adjoint(dat, spos, rpos), whole.nl_adjoint(dat, spos, rpos)
    else:
        sig = random_signals(spos, nts, rng)
        got, ref = sl.nl_forward(sig, spos, rpos), whole.nl_forward(sig, spos, rpos)
    assert max(np.abs(x).max() for x in ref) > 0
    _equal(got, ref)
    sl.close()
    whole.close()


def test_checkpoints_after_a_plan_that_ran_out_of_memory():
    """A change of storage that found no memory for all its states is not taken for a plan in place: the
    next forward makes the buffers that are missing."""
    nz, nx, ny, nts = 72, 200, 400, 6
    rng = np.random.default_rng(16)
    med = _medium(nz, nx, ny)
    sets = sp, so, rp, ro, sig = _device_sets(rng, nz, nx, ny, nts)
    out = []
    for short in (False, True):
        pr = _propagator(nz, nx, ny, nts)
        pr.set_medium(med)
        pr.set_velocity_storage("fp32")
        if short:
            rec = torch.empty((nts, ro[9]), device="cuda")
            pr.synchronize()
            with _memory_left(1.15 * 18 * 4 * nz * nx * ny):
                pr.step_only(0, 1)  # in unpadded rows from here on
                pr.synchronize()
            pr.set_checkpoint_policy("fp16", 2)
            pr.fwi_forward_device(sp, so, rp, ro, sig, rec)
            pr.synchronize()
            pr.set_checkpoint_policy("fp32", 2)
            with _memory_left(8 << 20):
                with pytest.raises(N.E3DError, match="memory"):
                    pr.fwi_forward_device(sp, so, rp, ro, sig, rec)
                torch.cuda.synchronize()
        pr.set_checkpoint_policy("fp32", 2)
        out.append(_gradient(pr, sets, nts, ny, nx, nz))
        assert pr.checkpoint_type == "fp32"
        pr.close()
    _equal(out[1], out[0])
