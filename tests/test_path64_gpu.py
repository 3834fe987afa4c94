"""The FP64 path over tiles (per-point fields, emitter chains, segments,
sums) against the allocation-free entry point's kernel, one thread per (ray,
channel) in the order of formod_pencil (jurassic.c:3196-3338): batches around
the tile size of 32 rays, both emissivity approximations, one to five
emitters, small batches (four lanes per ray) and larger ones (one), p-T grids
that differ between channels, rows that are not monotone, missing tables.

Tolerance: both forms round every table interpolation and path product
alike; only the continuum's factors are grouped differently, which moves a
segment's transmittance by at most a few units of 2^-53.  Over at most 2000
segments that is below 1e-12 of the path's emissivity scale; radiances are
compared to 1e-11."""
import ctypes as C

import numpy as np
import pytest

from jurassic_gb300 import native, synth
from test_zz_no_alloc import DeviceBatch

pytestmark = pytest.mark.gpu

RTOL = 1e-11


def _run(ctx, batch, entry):
    L = native.load()
    db = DeviceBatch(L, batch)
    try:
        db.reset_outputs()
        s = db.struct()
        rc = (L.jgb_formod_batch_dev(ctx.h, C.byref(s), native.FP64) if entry == "tiles"
              else L.jgb_formod_batch_dev_noalloc(ctx.h, C.byref(s)))
        assert rc == 0, L.jgb_last_error(ctx.h).decode()
        return db.outputs()
    finally:
        db.free()


def _compare(ctx, batch):
    a, b = _run(ctx, batch, "tiles"), _run(ctx, batch, "threads")
    for k in ("rad", "tau"):
        assert np.array_equal(np.isfinite(a[k]), np.isfinite(b[k])), k
        f = np.isfinite(b[k])
        scale = np.maximum(np.abs(b[k][f]), 1e-12 * np.max(np.abs(b[k][f])))
        assert np.max(np.abs(a[k][f] - b[k][f]) / scale) <= RTOL, k


@pytest.mark.parametrize("formod,nobs,nd,gases", [(1, 1, 2, 1), (0, 31, 5, 2), (1, 32, 3, 5),
                                                  (1, 33, 9, 3), (0, 70, 40, 4), (1, 130, 37, 2)])
def test_tiles_match_threads(built_lib, formod, nobs, nd, gases):
    w = synth.config_nadir(nobs, nd=nd, nlev=41, ztop=60.0, formod=formod,
                           emitters=("CO2", "H2O", "O3", "CH4", "N2O")[:gases])
    ctx = native.Context(w.ctl, w.tables, w.filters)
    b = w.batch.fresh_outputs()
    b.rad[0, ::3] = np.nan
    _compare(ctx, b)
    ctx.close()


@pytest.mark.parametrize("formod", [1, 0])
@pytest.mark.parametrize("what", ["grids", "rows", "missing", "limb"])
def test_tables_outside_the_usual_form(built_lib, formod, what):
    if what == "limb":
        w = synth.config_limb_ega(n_rays=35, formod=formod)
    else:
        w = synth.config_nadir(40, nd=6, nlev=31, ztop=50.0, formod=formod,
                               emitters=("CO2", "H2O", "O3"))
    t = w.tables
    if what == "grids":      # one channel's pressure grid differs
        t.p[2, 1] *= 1.003
        t.t[4, 0] += 0.25
    elif what == "rows":     # a column density that falls along a row
        n = int(t.nu[1, 0, 20, 15])
        t.u[1, 0, 20, 15, n // 2] = t.u[1, 0, 20, 15, n // 2 - 2]
    elif what == "missing":  # tables absent, pressures without temperatures
        t.np_[0, 1] = -1
        t.np_[3, :] = -1
        t.nt[:, 2, 5] = 1
    ctx = native.Context(w.ctl, t, w.filters)
    _compare(ctx, w.batch.fresh_outputs())
    ctx.close()


def test_batch_in_several_chunks(built_lib):
    """A batch whose workspaces exceed one chunk: its observations equal, bit
    for bit, the same ones in a smaller batch."""
    w = synth.config_nadir(800, nd=100)
    ctx = native.Context(w.ctl, w.tables, w.filters)
    out = ctx.formod_batch(w.batch.fresh_outputs(), native.FP64)
    for i in (0, 399, 799):
        atm, obs = w.batch.item(w.ctl, i)
        one = ctx.formod(atm, obs, native.FP64)
        assert np.array_equal(one.rad[:, 0], out.rad[:, i])
        assert np.array_equal(one.tau[:, 0], out.tau[:, i])
    ctx.close()
