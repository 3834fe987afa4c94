"""Ray tracing with several lanes per ray and the points in their own kernel.

A batch's walks fill warps of eight (mixed) or four (FP64) rays and the points
run 128 at a time, so each observation of a batch is compared, bit for bit, with
the same observation traced alone: batch sizes that leave a warp's or a block's
last rays empty, emitters beyond the eight that the Curtis-Godson sums take at
once, extinction windows, clouds.  FP64 batches above 6144 rays are walked by
one lane per ray: their rays equal the eight-lane walk's.  Both forms do the same
operations in the same order, so nothing is left to a tolerance."""
import copy

import numpy as np
import pytest

from jurassic_gb300 import native, synth

pytestmark = pytest.mark.gpu

GASES = ("CO2", "H2O", "O3", "CH4", "N2O", "CO", "HNO3", "F11", "F12")


def _same_alone(ctx, ctl, batch, precision, which):
    out = ctx.formod_batch(batch.fresh_outputs(), precision)
    for i in which:
        atm, obs = batch.item(ctl, i)
        one = ctx.formod(atm, obs, precision)
        r0, r1 = batch.ray_off[i], batch.ray_off[i + 1]
        assert np.array_equal(one.rad, out.rad[:, r0:r1])
        assert np.array_equal(one.tau, out.tau[:, r0:r1])
        assert np.array_equal(np.stack([one.tpz, one.tplon, one.tplat]), out.tp[:, r0:r1])
        assert np.all(np.isfinite(one.rad))


@pytest.mark.parametrize("precision", [native.MIXED, native.FP64])
@pytest.mark.parametrize("formod,nobs,gases,view", [(1, 9, 2, "nadir"), (0, 17, 9, "nadir"),
                                                    (0, 5, 3, "limb"), (1, 3, 8, "limb")])
def test_batch_equals_single(built_lib, precision, formod, nobs, gases, view):
    w = synth.config_nadir(nobs, nd=3, nlev=33, ztop=48.0, formod=formod, emitters=GASES[:gases])
    ctl, b = copy.deepcopy(w.ctl), w.batch
    if view == "limb":   # tangent altitudes from 4 to 40 km
        b.geo[1], b.geo[4] = 800.0, np.linspace(4.0, 40.0, nobs)
        b.geo[6] = b.geo[3] + 27.0
        ctl.raydz = 0.5
    ctl.window = np.array([0, 0, 0], dtype=np.int32)
    b.k = np.full((ctl.nw, b.k.shape[1]), 2e-4)
    ctx = native.Context(ctl, w.tables, w.filters)
    _same_alone(ctx, ctl, b, precision, range(nobs))
    ctx.close()


@pytest.mark.parametrize("formod", [1, 0])
def test_fp64_walks_of_a_large_batch(built_lib, formod):
    n = 6145
    w = synth.config_nadir(n, nd=1, nlev=21, ztop=40.0, formod=formod, emitters=GASES[:3])
    ctl = copy.deepcopy(w.ctl)
    ctl.raydz = 0.5
    ctx = native.Context(ctl, w.tables, w.filters)
    _same_alone(ctx, ctl, w.batch, native.FP64, (0, 31, 32, 6143, n - 1))
    ctx.close()
