"""Row sweeps with short and long chunks (64 positions below 20M elements, 256
from there on) and small-G sweeps of few rows: coefficients and one-way clustered
SEs of two-way panels against dense numpy algebra, at rows below a chunk, groups
that cross many chunks, both sides of the 20M elements, and single blocks."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_estimate, fe_runtime_config
from fe_gpu_gb300.bin_io import fe_host_arrays

pytestmark = pytest.mark.gpu


def demean(M, g, G):
    n = np.maximum(np.bincount(g, minlength=G), 1)
    out = np.empty_like(M)
    for j in range(M.shape[1]):
        out[:, j] = M[:, j] - (np.bincount(g, M[:, j], G) / n)[g]
    return out


@pytest.mark.parametrize("cluster", [1, 2])
@pytest.mark.parametrize("n,G,k", [(60, 7, 2), (257, 70, 3), (4097, 700, 3), (38_001, 700, 5), (200_003, 70, 4),
                                   (3_333_333, 700, 5), (3_333_334, 700, 5)])
def test_chunks_match_dense(built, n, G, k, cluster):
    T = 5
    rng = np.random.default_rng(n + k)
    a, b = rng.integers(0, G, size=n), rng.integers(0, T, size=n)
    a[:G], b[:T] = np.arange(G), np.arange(T)
    W = rng.standard_normal((n, k)) + 0.3 * b[:, None]
    y = W @ np.linspace(-1.0, 1.5, k) + 0.1 * a / G + 0.2 * b + rng.standard_normal(n)
    host = fe_host_arrays(y=y.copy(), W=np.asfortranarray(W), Z=np.zeros((n, 0), order="F"),
                          fe_ids=np.asfortranarray(np.vstack([a, b]).astype(np.int32) + 1))
    cfg = fe_runtime_config(fe_tolerance=1e-12, fe_max_iterations=2000, cluster_fe_dims=[cluster])
    res = fe_gpu_estimate(cfg, None, host)
    assert res.converged
    # the dense form: both dimensions partialled out
    Z = demean((b[:, None] == np.arange(T - 1)).astype(float), a, G)  # the last one follows from the others
    M = demean(np.column_stack([y, W]), a, G)
    M -= Z @ np.linalg.solve(Z.T @ Z, Z.T @ M)
    Y, X = M[:, 0], M[:, 1:]
    Q = np.linalg.inv(X.T @ X)
    beta = Q @ (X.T @ Y)
    S = X * (Y - X @ beta)[:, None]
    g, Gc = (a, G) if cluster == 1 else (b, T)
    sums = np.column_stack([np.bincount(g, S[:, j], Gc) for j in range(k)])
    scale = (n - 1) / (n - k - 1) * Gc / (Gc - 1)
    se = np.sqrt(np.diag(scale * Q @ (sums.T @ sums) @ Q))
    # means left at 1e-12 of unit columns, sums of up to 3.3M terms: below 1e-9 of the coefficients' scale
    np.testing.assert_allclose(res.beta, beta, rtol=0, atol=1e-9)
    np.testing.assert_allclose(res.se, se, rtol=1e-7, atol=0)
