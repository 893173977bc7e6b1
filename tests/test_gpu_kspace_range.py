"""Block products and updates of the Krylov column store on entries of mixed
size: the error is bounded entry by entry, by the sum of |x_i y_i|, as that of
an FP64 sum, not only by the product of the norms.

Products: a chunk of 128 rows is off by at most 128 x 2^-53 of its sum of
|x_i y_i| (the bound of an FP64 sum of 128 terms), and at most 64 more
additions meet in an entry at these sizes: 2^-45 (256 x 2^-53).  Updates of m
columns: m + 24 units of 2^-53 of sum |v_a C_ab| (the FP64 bound and what the
fixed-point sums may add to it), and the roundings of W, 8 units."""
import numpy as np
import pytest

import shear_nnf_gb300 as sb  # noqa: F401
from shear_nnf_gb300 import krylov as kr

pytestmark = pytest.mark.gpu


def _space(X):
    ks = kr.KSpace(*X.shape)
    for j in range(X.shape[1]):
        ks.set(j, X[:, j])
    return ks


def _products_within(X, m):
    p = X.shape[1] - m
    C = _space(X).gram(0, m, m, p)
    L = X.astype(np.longdouble)
    A, B = L[:, :m], L[:, m:]
    for j in range(p):
        t = A * B[:, j:j + 1]
        tol = 2.0 ** -45 * np.abs(t).sum(0)
        assert (np.abs(C[:, j] - t.sum(0)) <= tol).all(), (j, np.abs(C[:, j] - t.sum(0)) / tol)


@pytest.mark.parametrize("big", (1e4, 1e8, 1e12, 1e40))
@pytest.mark.parametrize("n,m,p", [(128, 4, 4), (131, 16, 1), (700, 9, 6), (4000, 70, 17)])
def test_products_of_large_entries_that_meet_zeros(n, m, p, big):
    """One large entry in every column and chunk of the left block, where the
    right block holds zeros."""
    rng = np.random.default_rng(n + m)
    X = rng.standard_normal((n, m + p))
    for c in range(0, n, 128):
        rows = c + rng.integers(0, min(128, n - c), 3)
        X[rows, m:] = 0.0
        X[rows[rng.integers(0, 3, m)], np.arange(m)] = big
    _products_within(X, m)


@pytest.mark.parametrize("n,m,p", [(128, 4, 4), (1000, 33, 5), (3000, 64, 16)])
def test_products_over_any_range(n, m, p):
    """Entries spread over forty orders of magnitude, each column its own way."""
    rng = np.random.default_rng(n)
    _products_within(rng.standard_normal((n, m + p)) * 10.0 ** rng.uniform(-20, 20, (n, m + p)), m)


def test_products_of_disjoint_and_zero_columns():
    """Supports that do not meet give exact zeros; zero columns too."""
    n, m, p = 640, 8, 4
    X = np.random.default_rng(1).standard_normal((n, m + p))
    X[::2, :m] = 0.0
    X[1::2, m:] = 0.0
    X[:, 3] = 0.0
    C = _space(X).gram(0, m, m, p)
    assert (C == 0.0).all()


def _update_within(X, m, M, alpha=1.0):
    p = X.shape[1] - m
    ks = _space(X)
    ks.update(0, m, m, p, M, alpha)
    L, LM = X.astype(np.longdouble), M.astype(np.longdouble)
    for b in range(p):
        t = L[:, :m] * LM[:, b]
        W = L[:, m + b] + np.longdouble(alpha) * t.sum(1)
        tol = 2.0 ** -53 * ((m + 24) * abs(alpha) * np.abs(t).sum(1) + 8 * np.abs(L[:, m + b])
                            + 2 * np.abs(W))
        err = np.abs(ks.get(m + b) - W)
        assert (err <= tol).all(), (b, float((err / np.maximum(tol, 1e-300)).max()))


@pytest.mark.parametrize("m,p", [(16, 1), (4, 4), (20, 3), (17, 16), (48, 33), (130, 8)])
@pytest.mark.parametrize("start", (0.0, 1.0))
def test_updates_of_entries_of_mixed_size(m, p, start):
    """Coefficients that pick single columns out of rows that hold numbers of
    every size, and full ones over many orders; W zero or not."""
    rng = np.random.default_rng(m + p)
    n = 900
    X = rng.standard_normal((n, m + p)) * 10.0 ** rng.uniform(-15, 15, (n, m + p))
    X[:, m:] = start * rng.standard_normal((n, p)) * 10.0 ** rng.uniform(-25, 5, (n, p))
    pick = np.zeros((m, p))
    pick[np.arange(m), np.arange(m) % p] = rng.choice([-1.0, 1.0, 3.0], m)
    _update_within(X, m, pick, -1.0)
    _update_within(X, m, rng.standard_normal((m, p)) * 10.0 ** rng.uniform(-12, 0, (m, p)), 0.5)
    _update_within(rng.standard_normal((n, m + p)), m, rng.standard_normal((m, p)), -0.75)


def test_updates_round_once():
    """130 columns: three parts of 0.3 units in the last place of W each give
    0.9, rounded to one."""
    m, p, n = 130, 2, 256
    X = np.zeros((n, m + p))
    X[:, [0, 64, 128]] = 0.3 * 2.0 ** -52
    X[:, m:] = 1.0
    ks = _space(X)
    ks.update(0, m, m, p, np.ones((m, p)), 1.0)
    for b in range(p):
        assert (ks.get(m + b) == 1.0 + 2.0 ** -52).all()
