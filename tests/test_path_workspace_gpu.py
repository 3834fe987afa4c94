"""Device memory of the path's workspaces (jgb_set_path_workspace).

Smaller workspaces cut a batch into more chunks of tiles and channels and change no
result: FP64 and mixed, EGA and CGA, reflecting surfaces, Jacobians resumed from their
bases and plain, bit for bit.  The workspaces keep to the limit, also for a batch
whose rays have no points (each tile then costs only its channels' words).  Where the
device has no room, the call gives back what it holds, goes on with a smaller limit,
which stays, and returns the same bits."""
import copy
import ctypes

import numpy as np
import pytest

from jurassic_gb300 import native, synth

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _surface(w):
    ctl = copy.deepcopy(w.ctl)
    ctl.sfnu, ctl.sftype = np.array([600.0, 2500.0]), 2
    w.batch.scal = np.zeros((w.batch.nobs, 5 + ctl.ncl + ctl.nsf))
    w.batch.scal[:, 4] = 288.0
    w.batch.scal[:, 5:] = 0.9
    return ctl


@pytest.mark.parametrize("formod", [1, 0])
@pytest.mark.parametrize("prec", [native.MIXED, native.FP64])
def test_forward_model_in_small_workspaces(built_lib, prec, formod):
    w = synth.config_nadir(200, nd=7, nlev=41, ztop=60.0, formod=formod, emitters=("CO2", "H2O", "O3"))
    ctx = native.Context(_surface(w), w.tables, w.filters)
    ref = ctx.formod_batch(w.batch.fresh_outputs(), prec)
    for limit in (MIB, 8 * MIB):
        ctx.set_path_workspace(limit)
        for split in (0, 1):
            ctx.set_path_split(split)
            out = ctx.formod_batch(w.batch.fresh_outputs(), prec)
            assert np.array_equal(out.rad, ref.rad) and np.array_equal(out.tau, ref.tau)
    assert ctx.path_workspace()[0] == 8 * MIB
    ctx.set_path_workspace(0)
    assert ctx.path_workspace()[0] == 4096 * MIB
    with pytest.raises(native.JurassicError):
        ctx.set_path_workspace(MIB - 1)
    ctx.close()


@pytest.mark.parametrize("formod", [1, 0])
def test_jacobians_in_small_workspaces(built_lib, formod):
    w = synth.config_nadir(40, nd=9, nlev=31, ztop=60.0, formod=formod, emitters=("CO2", "H2O", "O3"))
    ctl = copy.deepcopy(w.ctl)
    ctl.rett_zmin, ctl.rett_zmax = 10.0, 40.0
    ctl.retq_zmin, ctl.retq_zmax = np.array([-999.0, 0.0, 10.0]), np.array([-999.0, 20.0, 30.0])
    ctx = native.Context(ctl, w.tables, w.filters)
    ref = ctx.kernel_batch(w.batch.fresh_outputs(), native.MIXED)[0]
    for limit, mode in ((MIB, 2), (MIB, 0), (16 * MIB, 2)):
        ctx.set_path_workspace(limit)
        ctx.set_fd_resume(mode)
        for a, b in zip(ref, ctx.kernel_batch(w.batch.fresh_outputs(), native.MIXED)[0]):
            assert np.array_equal(a, b)
    ctx.close()


@pytest.mark.parametrize("prec", [native.MIXED, native.FP64])
def test_rays_without_points_keep_to_the_limit(built_lib, prec):
    """20000 rays that pass above the atmosphere (view point at 200 km), one in
    five thousand that does not: 625 tiles x 40 channels of stop words alone are 6.4
    MB and more."""
    w = synth.config_nadir(20000, nd=40, nlev=11, ztop=60.0, emitters=("CO2", "H2O"))
    b = w.batch
    b.geo[4] = np.where(np.arange(b.nobs) % 5000 == 7, 0.0, 200.0)
    ctx = native.Context(w.ctl, w.tables, w.filters)
    ref = ctx.formod_batch(b.fresh_outputs(), prec)
    ctx.set_path_workspace(2 * MIB)
    fields = 600 * 32 * 8 * 40     # a tile's points: at most 600, 40 doubles of fields
    out = ctx.formod_batch(b.fresh_outputs(), prec)
    held = ctx.path_workspace()[1]
    ctx.close()
    assert np.array_equal(out.rad, ref.rad) and np.array_equal(out.tau, ref.tau)
    # the limit or one tile's workspace in one channel, the fields of a tile, an eighth more
    assert held <= 1.125 * (2 * MIB + 8 * fields)


def _free_bytes():
    rt = ctypes.CDLL("libcudart.so.13")
    free, total = ctypes.c_size_t(0), ctypes.c_size_t(0)
    assert rt.cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def test_no_room_on_the_device(built_lib):
    """700 MB left: a call whose workspaces would take more (FP64 2.9 GB, mixed 1.0)
    takes a smaller limit and keeps it."""
    L = native.load()
    w = synth.config_nadir(500, nd=100, nlev=41, ztop=100.0)
    ctx = native.Context(w.ctl, w.tables, w.filters)
    ref = [ctx.formod_batch(w.batch.fresh_outputs(), p) for p in (native.FP64, native.MIXED)]
    held = ctx.path_workspace()[1]
    ctx.set_path_workspace(0)
    assert held > 2500 * MIB and ctx.path_workspace()[1] == 0
    z = np.linspace(0, 60, 1000)
    spd = np.exp(-np.abs(z[:, None] - z[None, :]) / 3.0)
    block = L.jgb_dev_alloc(_free_bytes() - 700 * MIB)
    assert block
    try:
        out = [ctx.formod_batch(w.batch.fresh_outputs(), p) for p in (native.FP64, native.MIXED, native.FP64)]
        limit, held = ctx.path_workspace()
        # inverses of 20 matrices of 1000 x 1000: 160 MB and 320 MB of scratch, for
        # which the workspaces make room
        inv, st = ctx.matrix_invert([spd] * 20)
        after = ctx.path_workspace()[1]
    finally:
        L.jgb_dev_free(ctypes.c_void_p(block))
    ctx.close()
    for a, b in zip(out, ref + ref[:1]):
        assert np.array_equal(a.rad, b.rad) and np.array_equal(a.tau, b.tau)
    assert 64 * MIB <= limit <= 512 * MIB
    assert held > 200 * MIB and after < held and not np.any(st)
    assert np.max(np.abs(inv[-1] @ spd - np.eye(1000))) < 1e-9
