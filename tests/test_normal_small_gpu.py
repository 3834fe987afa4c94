"""FP64 normal equations of problems with few columns: sizes around the 32 columns
and 32 rows of a block's tile, in one ragged batch, against numpy (relative 1e-12,
the bound of the FP64 path), and a cost that follows the size (4000 problems of 300
x 8 take less than 0.6 of the time of as many of 300 x 32, whose products are 13
times as many; padded to a tile they take the same)."""
import ctypes

import numpy as np
import pytest

from jurassic_gb300 import native, synth

pytestmark = pytest.mark.gpu


def _context():
    return native.Context(synth.config_limb_ega(n_rays=1).ctl)


def test_sizes_around_a_tile(built_lib):
    rng = np.random.default_rng(43)
    sizes = [(m, n) for m in (1, 2, 31, 32, 33, 65, 200) for n in (1, 2, 3, 7, 16, 31, 32, 33, 64)]
    Ks = [rng.standard_normal(s) * np.exp(rng.uniform(-3, 3, s[1]))[None, :] for s in sizes]
    ws = [np.exp(rng.uniform(-1, 1, m)) for m, _ in sizes]
    dys = [rng.standard_normal(m) for m, _ in sizes]
    ctx = _context()
    As, bs = ctx.normal_equations(Ks, ws, dys, native.FP64)
    ctx.close()
    for K, w, dy, A, b in zip(Ks, ws, dys, As, bs):
        X = K * w[:, None]
        Ar, br = X.T @ X, K.T @ (dy * w * w)
        d = np.sqrt(np.diag(Ar))
        assert np.max(np.abs(A - Ar) / np.outer(d, d)) <= 1e-12
        assert np.allclose(b, br, rtol=1e-10, atol=1e-12 * np.max(np.abs(br)))
        assert np.array_equal(A, A.T)


def _kernel_ms(ctx, m, n, count):
    L = native.load()
    rng = np.random.default_rng(n)
    ip = lambda v: v.ctypes.data_as(ctypes.POINTER(ctypes.c_int))  # noqa: E731
    dev = []
    for a in (rng.standard_normal(count * m * n), np.ones(count * m), np.ones(count * m),
              np.zeros(count * n * n), np.zeros(count * n)):
        dev.append(ctypes.c_void_p(L.jgb_dev_alloc(a.nbytes)))
        assert L.jgb_memcpy_h2d(dev[-1], a.ctypes.data_as(ctypes.c_void_p), a.nbytes) == 0
    ms, best = ctypes.c_float(), 1e30
    ms_, ns_ = np.full(count, m, np.int32), np.full(count, n, np.int32)
    for _ in range(5):
        ctx._check(L.jgb_normal_equations_dev(ctx.h, count, ip(ms_), ip(ns_), *dev, native.FP64,
                                              ctypes.byref(ms)))
        best = min(best, ms.value)
    for p in dev:
        L.jgb_dev_free(p)
    return best


def test_cost_follows_the_columns(built_lib):
    ctx = _context()
    few, tile = _kernel_ms(ctx, 300, 8, 4000), _kernel_ms(ctx, 300, 32, 4000)
    ctx.close()
    assert few < 0.6 * tile, (few, tile)
