"""Accuracy of the batched matrix_invert in 64 bits, against inverses refined in
long double.

The yardstick is a plain Cholesky inverse by columns in the same 64 bits whose
sums are formed apart and subtracted once.  The errors of two such orders of
summation differ by tens of per cent from matrix to matrix and by less in the
mean over a set; an order that subtracts the products one by one from entries of
the matrix's size is 2.2 to 2.9 times as wrong on exponentially correlated
covariances.  The geometric mean of the errors' ratio over a set of matrices stays
below 1.5, between the two."""
import numpy as np
import pytest

from jurassic_gb300 import native, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


def _plain_inverse(a):
    n = len(a)
    L = np.zeros((n, n))
    for j in range(n):
        v = a[j:, j] - L[j:, :j] @ L[j, :j]
        L[j, j] = np.sqrt(v[0])
        L[j + 1:, j] = v[1:] / L[j, j]
    x = np.eye(n)
    for i in range(n):
        x[i] = (x[i] - L[i, :i] @ x[:i]) / L[i, i]
    for i in range(n - 1, -1, -1):
        x[i] = (x[i] - L[i + 1:, i] @ x[i + 1:]) / L[i, i]
    return 0.5 * (x + x.T)


def _refined_inverse(a):
    x = np.linalg.inv(a).astype(np.longdouble)
    for _ in range(3):
        r = np.eye(len(a), dtype=np.longdouble) - a.astype(np.longdouble) @ x
        x = x + (x.astype(np.float64) @ r.astype(np.float64))
    return x


@pytest.mark.parametrize("sizes", [(5, 12, 20, 27, 32, 8, 30, 17), (40, 53, 64, 70, 86, 100, 131, 150)])
@pytest.mark.parametrize("kind", ["covariance", "gauss-newton"])
def test_errors_no_larger_than_a_plain_inverse(built_lib, kind, sizes):
    rng = np.random.default_rng(31)
    mats = []
    for n in sizes:
        if kind == "covariance":
            z = np.linspace(0, 60, n)
            sd = 1.5 + 0.3 * np.clip(rng.standard_normal(n), -3, 3)
            mats.append(sd[:, None] * sd[None, :] * np.exp(-np.abs(z[:, None] - z[None, :]) / 3.0))
        else:
            b = rng.standard_normal((n, n))
            mats.append(b @ b.T / n + 0.5 * np.eye(n))
    ctx = native.Context(synth.config_nadir(1, nd=2, nlev=11).ctl)
    inv, st = ctx.matrix_invert(mats)
    ctx.close()
    assert not np.any(st)
    ratio = []
    for a, g in zip(mats, inv):
        x = _refined_inverse(a)
        err = [float(np.sqrt(np.sum((y - x) ** 2))) for y in (g, _plain_inverse(a))]
        ratio.append(err[0] / err[1])
    assert np.exp(np.mean(np.log(ratio))) <= 1.5, ratio


@pytest.mark.parametrize("n,at", [(6, 2), (32, 31), (40, 5), (70, 40)])
def test_infinite_variance(built_lib, built_oracle, n, at):
    """An element without any a-priori knowledge (infinite variance) has zero
    precision; the others' inverse is that of the matrix without it."""
    z = np.linspace(0, 60, n)
    a = 4.0 * np.exp(-np.abs(z[:, None] - z[None, :]) / 8.0)
    a[at, at] = np.inf
    ref, ok = oracle.matrix_invert(a)
    ctx = native.Context(synth.config_nadir(1, nd=2, nlev=11).ctl)
    inv, st = ctx.matrix_invert([a])
    ctx.close()
    assert ok and st[0] == 0
    assert np.all(inv[0][at] == 0) and np.all(inv[0][:, at] == 0)
    assert np.max(np.abs(inv[0] - ref)) <= 1e-10 * np.max(np.abs(ref))
