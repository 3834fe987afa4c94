"""Emitters without a column and profiles with values that are not numbers.

In the Curtis-Godson approximation an emitter without a column has no mean pressure
or temperature (0 / 0): it adds nothing, in FP64 as in the mixed path and in the
allocation-free entry point.  The radiances with a gas that is absent everywhere
equal those of a control set without its table, and the two precisions agree within
10 mK.  A mixing ratio that is not a number reaches the radiances of its own
observation, and only those."""
import copy

import numpy as np
import pytest

from jurassic_gb300 import native, synth
from jurassic_gb300.model import brightness

pytestmark = pytest.mark.gpu


def _bt_diff(a, b, nu):
    return np.max(np.abs(brightness(a, nu) - brightness(b, nu)))


@pytest.mark.parametrize("nobs", [5, 70])          # four lanes per ray and one in FP64: 0.2 and 2.4 warps per SM
@pytest.mark.parametrize("above", [-1.0, 20.0])    # absent everywhere, above 20 km
def test_absent_gas_adds_nothing_in_cga(built_lib, above, nobs):
    w = synth.config_nadir(nobs, nd=40, nlev=26, ztop=50.0, formod=0, emitters=("CO2", "N2O", "O3"))
    b = w.batch
    b.q[1] = np.where(b.z > above, 0.0, b.q[1])
    ctx = native.Context(w.ctl, w.tables, w.filters)
    f64 = ctx.formod_batch(b.fresh_outputs(), native.FP64)
    mix = ctx.formod_batch(b.fresh_outputs(), native.MIXED)
    ctx.close()
    nu = np.asarray(w.ctl.nu)[:, None]
    assert np.all(np.isfinite(f64.rad)) and np.all(f64.rad > 0)
    assert _bt_diff(f64.rad, mix.rad, nu) <= 0.010
    if above < 0:
        t = copy.deepcopy(w.tables)
        t.np_[:, 1] = -1
        ctx = native.Context(w.ctl, t, w.filters)
        without = ctx.formod_batch(b.fresh_outputs(), native.FP64)
        ctx.close()
        assert np.max(np.abs(f64.rad - without.rad) / without.rad) <= 1e-9


@pytest.mark.parametrize("formod", [1, 0])
@pytest.mark.parametrize("prec", [native.FP64, native.MIXED])
def test_mixing_ratio_that_is_not_a_number(built_lib, prec, formod):
    w = synth.config_nadir(5, nd=4, nlev=26, ztop=50.0, formod=formod, emitters=("CO2", "H2O", "O3"))
    b = w.batch
    b.q[0, b.lev_off[1] + 7] = np.nan              # CO2, with a continuum in every channel
    ctx = native.Context(w.ctl, w.tables, w.filters)
    out = ctx.formod_batch(b.fresh_outputs(), prec)
    ctx.close()
    assert np.all(np.isnan(out.rad[:, 1]))
    assert np.all(np.isfinite(np.delete(out.rad, 1, axis=1)))
