"""matrix_invert at the edges of its 32 x 32 tiles, in one ragged batch, against
the oracle: FP64 within 1e-10 of the largest inverse entry (the factor's sums run
in another order; the matrices' condition numbers are below 1e3)."""
import numpy as np
import pytest

from jurassic_gb300 import native, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


def test_matrix_invert_tile_edges(built_lib, built_oracle):
    rng = np.random.default_rng(23)
    mats = []
    for n in (2, 31, 32, 33, 63, 64, 65, 96, 97, 129):
        b = rng.standard_normal((n, n))
        mats.append(b @ b.T / n + 0.5 * np.eye(n))
    bad = mats[3].copy()
    bad[32, 32] = -1.0                  # fails in the second tile
    mats.append(bad)
    w = synth.config_nadir(1, nd=2, nlev=11)
    ctx = native.Context(w.ctl, w.tables, w.filters)
    inv, st = ctx.matrix_invert(mats)
    for a, g, s in zip(mats, inv, st):
        ref, ok = oracle.matrix_invert(a)
        assert (s == 0) == ok
        if not ok:
            assert np.array_equal(g, a)  # left as it was
            continue
        assert np.max(np.abs(g - ref)) <= 1e-10 * np.max(np.abs(ref))
        assert np.array_equal(g, g.T)
    ctx.close()
