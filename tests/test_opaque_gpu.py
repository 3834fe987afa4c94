"""Opaque scenes of the mixed path: rays behind a thick cloud or a strong window
extinction end where the path is opaque.

The ends change no result: with them (one lane per ray) and without (four lanes)
the radiances and transmittances are the same bits, for clouds, extinctions, both,
negative and non-finite extinctions and reflecting surfaces; Jacobians resumed from
their bases equal the plain ones.  And the points behind them cost nothing: a
batch whose extinction begins at 80 of 100 km takes less than 0.6 of the clear
batch's path time (a fifth of the points, and what does not depend on them)."""
import copy

import numpy as np
import pytest

from jurassic_gb300 import native, synth

pytestmark = pytest.mark.gpu


def _scene(what, nobs=70, **kw):
    w = synth.config_nadir(nobs, nd=5, nlev=51, ztop=100.0, emitters=("CO2", "H2O", "O3"), **kw)
    ctl, b = copy.deepcopy(w.ctl), w.batch
    ctl.nw, ctl.window = 2, np.array([0, 0, 1, 1, 0], dtype=np.int32)
    ctl.retk_zmin = ctl.retk_zmax = np.full(2, -999.0)
    nl = b.nlev
    z = b.z
    b.k = np.zeros((2, nl))
    if what in ("cloud", "both", "surface"):
        ctl.clnu = np.array([600.0, 2500.0])
    if what == "surface":
        ctl.sfnu, ctl.sftype = np.array([600.0, 2500.0]), 2
    b.scal = np.zeros((nobs, 5 + ctl.ncl + ctl.nsf))
    if ctl.ncl:
        rng = np.random.default_rng(5)
        b.scal[:, 0] = rng.uniform(5, 60, nobs)
        b.scal[:, 1] = np.where(np.arange(nobs) % 3, rng.uniform(0.5, 8.0, nobs), 0.0)
        b.scal[:, 2:4] = 10.0 ** rng.uniform(-2, 1.5, (nobs, 2))
    if ctl.nsf:
        b.scal[:, 4 + ctl.ncl] = 285.0
        b.scal[:, 5 + ctl.ncl:] = np.where(np.arange(nobs) % 2, 0.9, 1.0)[:, None]
    lev = np.arange(nl) % 51
    if what in ("extinction", "both"):
        b.k[0] = np.where(z < 40, 3.0, 0.0)
        b.k[1] = np.where(z < 70, np.exp(-z / 10.0), 0.0)
    if what == "negative":
        b.k[0] = np.where(z < 60, 4.0, np.where(z < 90, -1.0, 0.0))
        b.k[1] = np.where(lev == 30, -50.0, 2.0)
    if what == "not finite":
        b.k[0] = np.where(z < 60, 4.0, 0.0)
        b.k[0][lev == 20] = np.inf
        b.k[1] = 1.0
        b.k[1][lev == 10] = np.nan
    return w, ctl, b


@pytest.mark.parametrize("formod", [1, 0])
@pytest.mark.parametrize("what", ["cloud", "extinction", "both", "surface", "negative", "not finite"])
def test_ends_change_nothing(built_lib, what, formod):
    w, ctl, b = _scene(what, formod=formod)
    ctx = native.Context(ctl, w.tables, w.filters)
    out = []
    for split in (0, 1):
        ctx.set_path_split(split)
        out.append(ctx.formod_batch(b.fresh_outputs(), native.MIXED))
    ctx.close()
    for k in ("rad", "tau"):
        assert np.array_equal(getattr(out[0], k), getattr(out[1], k), equal_nan=True)
    if what != "not finite":
        assert np.all(np.isfinite(out[0].rad))


@pytest.mark.parametrize("what", ["cloud", "extinction", "negative"])
def test_resumed_jacobians_of_opaque_scenes(built_lib, what):
    w, ctl, b = _scene(what, nobs=6)
    ctl.rett_zmin, ctl.rett_zmax = 0.0, 80.0
    ctl.retq_zmin, ctl.retq_zmax = np.zeros(3), np.array([60.0, -999.0, 40.0])
    ctl.retk_zmin, ctl.retk_zmax = np.array([10.0, -999.0]), np.array([90.0, -999.0])
    ctx = native.Context(ctl, w.tables, w.filters)
    res = []
    for mode, split in ((2, 0), (2, 1), (0, 0), (0, 1)):
        ctx.set_fd_resume(mode)
        ctx.set_path_split(split)
        res.append(ctx.kernel_batch(b.fresh_outputs(), native.MIXED)[0])
    ctx.close()
    for other in res[1:]:
        for a, c in zip(res[0], other):
            assert np.array_equal(a, c) and np.all(np.isfinite(a))


def _path_ms(ctx, b, call):
    best = 1e30
    for _ in range(6):
        call(b.fresh_outputs())
        best = min(best, ctx.stats()["path_ms"])
    return best


def test_points_behind_an_opaque_layer_cost_nothing(built_lib):
    w = synth.config_nadir(6000, nd=20, nlev=51, ztop=100.0, emitters=("CO2", "H2O", "O3"))
    ctx = native.Context(w.ctl, w.tables, w.filters)
    call = lambda q: ctx.formod_batch(q, native.MIXED)  # noqa: E731
    clear = _path_ms(ctx, w.batch, call)
    w.batch.k[0] = np.where(w.batch.z < 80, 5.0, 0.0)
    opaque = _path_ms(ctx, w.batch, call)
    ctx.close()
    assert opaque < 0.6 * clear, (opaque, clear)
