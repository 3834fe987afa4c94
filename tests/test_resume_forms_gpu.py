"""Resumed Jacobians with tables outside the usual form: p-T grids that differ between
channels, rows that fall, tables and temperature rows that are missing.  The emitters'
kernel then searches the cell at every point and carries that search across a resume;
with few bases four lanes walk a base ray, with many one.  The Jacobians equal the
plain ones bit for bit, in EGA and CGA."""
import copy

import numpy as np
import pytest

from jurassic_gb300 import native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nobs,nd", [(6, 6), (1500, 21)])  # 1500: 47 tiles x 21 x 3 warps, above 18 per SM
@pytest.mark.parametrize("formod", [1, 0])
@pytest.mark.parametrize("what", ["grids", "rows", "missing"])
def test_resumed_equals_plain(built_lib, what, formod, nobs, nd):
    w = synth.config_nadir(nobs, nd=nd, nlev=26, ztop=50.0, formod=formod, emitters=("CO2", "H2O", "O3"))
    t = w.tables
    if what == "grids":      # one channel's pressure grid differs, one's temperatures
        t.p[2, 1] *= 1.003
        t.t[4, 0] += 0.25
    elif what == "rows":     # a column density that falls along a row
        n = int(t.nu[1, 0, 20, 15])
        t.u[1, 0, 20, 15, n // 2] = t.u[1, 0, 20, 15, n // 2 - 2]
    else:                    # tables absent, pressures without temperatures
        t.np_[0, 1] = -1
        t.np_[3, :] = -1
        t.nt[:, 2, 5] = 1
    ctl = copy.deepcopy(w.ctl)
    ctl.rett_zmin, ctl.rett_zmax = 11.0, 15.0                  # two levels each
    ctl.retq_zmin, ctl.retq_zmax = np.array([3.0, -999.0, 19.0]), np.array([7.0, -999.0, 23.0])
    ctx = native.Context(ctl, t, w.filters)
    ctx.set_fd_resume(0)
    plain = ctx.kernel_batch(w.batch.fresh_outputs(), native.MIXED)[0]
    ctx.set_fd_resume(2)
    resumed = ctx.kernel_batch(w.batch.fresh_outputs(), native.MIXED)[0]
    assert ctx.stats()["resume_skip"] > 0.05
    ctx.close()
    for a, b in zip(resumed, plain):
        assert np.array_equal(a, b) and np.all(np.isfinite(a))
