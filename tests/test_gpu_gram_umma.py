"""The tensor-core Gram at the edges of its tiles: block widths around 16
columns, rows around the tiles of 2048 / columns values and the 1024-row sums,
columns whose scale rises on the way, zeros, and values that are not finite."""
import numpy as np
import pytest

from fe_gpu_gb300 import _native as N

pytestmark = pytest.mark.gpu


def gram(X):
    X = np.ascontiguousarray(X, dtype=np.float64)
    n, a = X.shape
    out = np.zeros((a, a), order="F")
    N.check(N.lib().fegb_test_gram(X.ctypes.data, n, a, 1, out.ctypes.data), "fegb_test_gram")
    return out


@pytest.mark.parametrize("n,a", [(1, 1), (1025, 2), (17, 5), (223, 9), (4097, 9), (9000, 8), (1023, 15), (1024, 16),
                                 (1025, 17), (5000, 31), (129, 32), (3000, 33), (70_001, 6), (2000, 111)])
def test_whole_numbers_are_exact(built, n, a):
    """|x| <= 1000 in whole numbers: every sum is below 2^53, so every form of exact products and FP64 sums gives it"""
    X = np.random.default_rng(n + a).integers(-1000, 1001, size=(n, a)).astype(np.float64)
    np.testing.assert_array_equal(gram(X), X.T @ X)


@pytest.mark.parametrize("n,a", [(40_000, 40), (66_000, 9), (5_000, 17)])
def test_scales(built, n, a):
    rng = np.random.default_rng(a)
    X = rng.normal(size=(n, a)) * rng.uniform(1e-3, 1e3, size=a)
    X[:, 0] = 0.0
    X[:, 1] = rng.uniform(size=n) < 0.003  # rare ones
    X[: n // 2, 2] = 0.0
    X[: n // 2, 3] *= 1e-9
    X[:, 4] = rng.standard_cauchy(n)
    X[: n // 3, 5] *= 1e-290
    X[:, 6] *= 1e140
    X[:, 7] *= -1e-140
    X[:, 8] = -(2.0**58 + float(0x80808080808080)) * 2.0**-40  # seven digits of -128 below the first
    L = X.astype(np.longdouble)
    ref = (L.T @ L).astype(np.float64)
    got = gram(X)
    norm = np.sqrt(np.diag(ref))
    norm[norm == 0] = 1.0
    # digits: 2^-58 of a column's largest value, at most sqrt(n) 2^-57 of the norms;
    # fewer than 100 FP64 additions of partial sums at 2^-53 each
    tol = 100 * 2.0**-53 + np.sqrt(n) * 2.0**-57
    assert np.max(np.abs(got - ref) / norm[:, None] / norm[None, :]) < tol
    assert np.all(got[0] == 0.0)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_not_finite(built, value):
    X = np.random.default_rng(3).normal(size=(5000, 6))
    X[4321, 2] = value
    got = gram(X)
    with np.errstate(invalid="ignore"):
        ref = X.T @ X
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(np.isinf(got), np.isinf(ref))
    keep = np.isfinite(ref)
    np.testing.assert_allclose(got[keep], ref[keep], rtol=1e-12, atol=1e-9)
