"""Cloud extinctions that are not finite: both precisions treat them alike.

An extinction that is not a number (a NaN in the control vector, or two infinite
table entries, between which the interpolation has no value) makes the radiances
of the observations with a cloud not a number, and those only; an infinite one
makes the cloud black.  The finite radiances of the two precisions agree within
10 mK, the mixed path's bound."""
import copy

import numpy as np
import pytest

from jurassic_gb300 import native, synth
from jurassic_gb300.model import brightness

pytestmark = pytest.mark.gpu

NAN, INF = np.nan, np.inf


@pytest.mark.parametrize("lanes4", [0, 1])
@pytest.mark.parametrize("clk", [(NAN, 0.02), (NAN, NAN), (INF, INF), (0.02, INF), (0.02, 0.03)])
def test_cloud_extinction_not_finite(built_lib, clk, lanes4):
    w = synth.config_nadir(35, nd=5, nlev=31, ztop=60.0, emitters=("CO2", "H2O"))
    ctl = copy.deepcopy(w.ctl)
    ctl.clnu = np.array([600.0, 2500.0])   # every channel lies strictly between
    b = w.batch
    b.scal = np.zeros((b.nobs, 5 + ctl.ncl + ctl.nsf))
    b.scal[:, 0] = 9.0
    b.scal[::2, 1] = 20.0                  # every other observation has a cloud
    b.scal[:, 2:4] = clk
    ctx = native.Context(ctl, w.tables, w.filters)
    ctx.set_path_split(lanes4)
    mixed = ctx.formod_batch(b.fresh_outputs(), native.MIXED)
    ref = ctx.formod_batch(b.fresh_outputs(), native.FP64)
    ctx.close()
    bad = np.isnan(clk[0] + (clk[1] - clk[0]))
    for o in (mixed, ref):
        assert np.all(np.isnan(o.rad[:, ::2]) if bad else np.isfinite(o.rad[:, ::2]))
        assert np.all(np.isfinite(o.rad[:, 1::2]))
    nu = np.asarray(ctl.nu)[:, None]
    on = np.isfinite(ref.rad)
    d = np.abs(brightness(np.where(on, mixed.rad, 1.0), nu) - brightness(np.where(on, ref.rad, 1.0), nu))
    assert np.max(d) <= 0.010
