"""Forms of the mixed path's kernels beyond the usual tables and sizes.

Tables whose p-T grids differ between channels, whose rows are not monotone or
which are missing take the general emitters' kernel: four lanes per ray and one
give the same bits, and both stay within 10 mK of the FP64 path, the mixed path's
bound.  A Jacobian whose base segments exceed the path's workspace runs in
groups of channels: the same bits as the plain one."""
import copy

import numpy as np
import pytest

from jurassic_gb300 import native, synth
from jurassic_gb300.model import brightness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("formod", [1, 0])
@pytest.mark.parametrize("what", ["grids", "rows", "missing"])
def test_tables_outside_the_usual_form(built_lib, formod, what):
    w = synth.config_nadir(33, nd=6, nlev=31, ztop=50.0, formod=formod, emitters=("CO2", "H2O", "O3"))
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
    ctx = native.Context(w.ctl, t, w.filters)
    out = []
    for split in (0, 1):
        ctx.set_path_split(split)
        out.append(ctx.formod_batch(w.batch.fresh_outputs(), native.MIXED))
    assert np.array_equal(out[0].rad, out[1].rad) and np.array_equal(out[0].tau, out[1].tau)
    ref = ctx.formod_batch(w.batch.fresh_outputs(), native.FP64)
    nu = np.asarray(w.ctl.nu)[:, None]
    on = ref.rad > 0   # a channel without tables has continua only
    assert np.array_equal(on, out[0].rad > 0)
    d = np.abs(brightness(np.where(on, out[0].rad, 1.0), nu) - brightness(np.where(on, ref.rad, 1.0), nu))
    assert np.max(d) <= 0.010
    ctx.close()


def test_resumed_jacobian_in_channel_groups(built_lib):
    w = synth.config_nadir(3000, nd=60, nlev=31, ztop=100.0)
    ctl = copy.deepcopy(w.ctl)
    dz = 100.0 / 30
    ctl.rett_zmin, ctl.rett_zmax = 2.5 * dz, 4.5 * dz          # two levels
    ctl.retq_zmin = np.array([-999.0, 2.5 * dz, -999.0, -999.0, -999.0])
    ctl.retq_zmax = np.array([-999.0, 4.5 * dz, -999.0, -999.0, -999.0])
    ctx = native.Context(ctl, w.tables, w.filters)
    res = []
    for mode in (2, 0):
        ctx.set_fd_resume(mode)
        Ks, _ = ctx.kernel_batch(w.batch.fresh_outputs(), native.MIXED)
        res.append(Ks)
        if mode == 2:
            assert ctx.stats()["resume_skip"] > 0.05
    for a, c in zip(*res):
        assert np.array_equal(a, c) and np.all(np.isfinite(a))
    ctx.close()
