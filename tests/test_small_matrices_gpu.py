"""matrix_invert of small matrices: every size up to two tiles against the oracle,
in one ragged batch, and a cost that follows the size (20000 matrices of 2 x 2 take
less than 0.3 of the time of as many of 32 x 32, whose products are 4096 times as
many; padded to a tile they take more than half)."""
import ctypes

import numpy as np
import pytest

from jurassic_gb300 import native, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


def _context():
    return native.Context(synth.config_nadir(1, nd=2, nlev=11).ctl)


def test_every_small_size(built_lib, built_oracle):
    rng = np.random.default_rng(41)
    mats = []
    for n in list(range(1, 67)) * 2:
        b = rng.standard_normal((n, n))
        mats.append(b @ b.T / n + 0.5 * np.eye(n))
    for n, at in ((2, 1), (9, 0), (32, 31), (33, 32), (64, 40)):  # not positive definite
        a = mats[n - 1].copy()
        a[at, at] = -1.0
        mats.append(a)
    ctx = _context()
    inv, st = ctx.matrix_invert(mats)
    ctx.close()
    for a, g, s in zip(mats, inv, st):
        ref, ok = oracle.matrix_invert(a)
        assert (s == 0) == ok
        if not ok:
            assert np.array_equal(g, a)
            continue
        assert np.max(np.abs(g - ref)) <= 1e-10 * np.max(np.abs(ref))
        assert np.array_equal(g, g.T)


def _kernel_ms(ctx, n, count):
    L = native.load()
    rng = np.random.default_rng(n)
    b = rng.standard_normal((count, n, n))
    a = np.ascontiguousarray(b @ b.transpose(0, 2, 1) / n + 0.5 * np.eye(n))
    sizes = np.full(count, n, np.int32)
    dev = ctypes.c_void_p(L.jgb_dev_alloc(a.nbytes))
    ms, best = ctypes.c_float(), 1e30
    for _ in range(5):
        assert L.jgb_memcpy_h2d(dev, a.ctypes.data_as(ctypes.c_void_p), a.nbytes) == 0
        ctx._check(L.jgb_matrix_invert_dev(ctx.h, count, sizes.ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
                                           dev, None, ctypes.byref(ms)))
        best = min(best, ms.value)
    L.jgb_dev_free(dev)
    return best


def test_cost_follows_the_size(built_lib):
    ctx = _context()
    small, tile = _kernel_ms(ctx, 2, 20000), _kernel_ms(ctx, 32, 20000)
    ctx.close()
    assert small < 0.3 * tile, (small, tile)
