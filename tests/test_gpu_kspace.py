"""Block products and block updates of the Krylov column store at the edges of
their tiles: columns of any scale, zero columns, infinities and NaN, row
ranges, against extended precision.  The fixed-point sums keep 58 bits of a
chunk's largest entry; over at most 256 rows the rounded digits of one side
weigh up to 2^-59 sqrt(256) |x| max|y|, both sides and the dropped product
2^-53 |x| |y|, and the sums of the chunks a few 2^-53 more: 2^-51 |x| |y|.
An update of m <= 64 columns rounds each product at 2^-57 of the row's largest
scaled entry times the largest scaled coefficient, and once more at the end."""
import numpy as np
import pytest

import shear_nnf_gb300 as sb
from shear_nnf_gb300 import krylov as kr

pytestmark = pytest.mark.gpu


def _fill(ks, X):
    for j in range(X.shape[1]):
        ks.set(j, X[:, j])


def _columns(n, cols, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, cols)) * np.exp(-rng.uniform(0, 12, (n, 1)))
    X *= 10.0 ** rng.integers(-30, 30, cols)
    X[:, 1] = 0.0
    X[: n // 2, 3] = 0.0
    return X


@pytest.mark.parametrize("n,m,p,lo,hi", [
    (1, 4, 4, 0, 1), (63, 5, 4, 1, 62), (64, 16, 1, 0, 64), (255, 17, 3, 0, 255),
    (257, 64, 16, 0, 257), (2000, 65, 17, 3, 1999), (5000, 7, 33, 0, 5000), (90000, 20, 5, 11, 89999)])
def test_products_and_updates(n, m, p, lo, hi):
    X = _columns(n, m + p, n + m + p)
    ks = kr.KSpace(n, m + p)
    _fill(ks, X)
    L = X.astype(np.longdouble)
    A, B = L[lo:hi, :m], L[lo:hi, m:]
    C = ks.gram(0, m, m, p, rows=(lo, hi))
    nrm = np.sqrt((A * A).sum(0))[:, None] * np.sqrt((B * B).sum(0))
    ref = np.stack([(A * B[:, j:j + 1]).sum(0) for j in range(p)], axis=1)
    assert (np.abs(C - ref) <= 2.0 ** -51 * nrm).all()
    assert np.array_equal(ks.gram(0, m, m, p, rows=(lo, hi)), C)

    M = np.random.default_rng(7).standard_normal((m, p))
    M[0] *= 1e12
    M[:, 0] *= 1e-20
    M[m // 2] = 0.0
    ks.update(0, m, m, p, M, -0.75, rows=(lo, hi))
    W = L[:, m:].copy()
    W[lo:hi] -= 0.75 * np.stack([(A * M[:, j].astype(np.longdouble)).sum(1) for j in range(p)],
                                axis=1)
    tol = 2.0 ** -52 * np.abs(W)
    for c in range(0, m, 64):
        s = np.abs(M[c:c + 64]).max(1)
        big = (np.abs(A[:, c:c + 64]) * s).max(1)[:, None] * 2
        rel = np.divide(np.abs(M[c:c + 64]), s[:, None], where=s[:, None] > 0,
                        out=np.zeros_like(M[c:c + 64])).max(0) * 2
        tol[lo:hi] += 2.0 ** -51 * big * rel + 2.0 ** -52 * np.abs(W[lo:hi])
    got = np.stack([ks.get(m + j) for j in range(p)], axis=1)
    assert (np.abs(got - W) <= tol).all()
    assert np.array_equal(got[:lo], X[:lo, m:]) and np.array_equal(got[hi:], X[hi:, m:])
    for j in range(m):
        assert np.array_equal(ks.get(j), X[:, j])


@pytest.mark.parametrize("value", [np.inf, np.nan, 1e200, 1e-310])
def test_values_outside_the_fixed_point_range(value):
    n, m, p = 700, 9, 6
    X = np.random.default_rng(3).standard_normal((n, m + p))
    X[300, 2] = value
    X[5, m + 1] = value
    ks = kr.KSpace(n, m + p)
    _fill(ks, X)
    with np.errstate(all="ignore"):
        ref = X[:, :m].T @ X[:, m:]
        C = ks.gram(0, m, m, p)
        np.testing.assert_allclose(C, ref, rtol=1e-12, atol=1e-12)
        M = np.random.default_rng(4).standard_normal((m, p))
        ks.update(0, m, m, p, M, 1.0)
        got = np.stack([ks.get(m + j) for j in range(p)], axis=1)
        np.testing.assert_allclose(got, X[:, m:] + X[:, :m] @ M, rtol=1e-12, atol=1e-12)
        M[3, 2] = value
        _fill(ks, X)
        ks.update(0, m, m, p, M, 1.0)
        got = np.stack([ks.get(m + j) for j in range(p)], axis=1)
        np.testing.assert_allclose(got, X[:, m:] + X[:, :m] @ M, rtol=1e-12, atol=1e-12)
