"""Runs of rows with equal ids as the operator's tuples: pairs of several runs
(merged for clusters over both dimensions), and runs given up because pairs come
back too often, which cost no memory for the rest of the call."""
import ctypes as C

import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_estimate, fe_gpu_within_transform, fe_runtime_config
from fe_gpu_gb300 import _native as N
from fe_gpu_gb300.bin_io import fe_host_arrays
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def panel(workers, firms, years, pattern, seed):
    """Workers of len(pattern) rows; pattern[t]: which of the worker's firms in row t"""
    rng = np.random.default_rng(seed)
    pattern = np.asarray(pattern)
    own = np.stack([rng.choice(firms, pattern.max() + 1, replace=False) for _ in range(workers)])
    w = np.repeat(np.arange(workers), len(pattern))
    f = own[w, np.tile(pattern, workers)]
    ids = [w, f] + ([rng.integers(0, years, len(w))] if years else [])
    W = rng.standard_normal((len(w), 3)) + 0.3 * rng.standard_normal(firms)[f][:, None]
    y = W @ np.array([0.5, -0.3, 0.2]) + rng.standard_normal(firms)[f] + rng.standard_normal(workers)[w] \
        + rng.standard_normal(len(w))
    return y, np.asfortranarray(W), np.asfortranarray(np.vstack(ids).astype(np.int32) + 1)


def host(y, W, fe):
    return fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((len(y), 0), order="F"), fe_ids=fe)


# 11 runs a worker in 10 pairs: merged; 10 runs in 2 pairs: given up; 21 runs, the pairs of the first 17 back after
# more runs than are looked at: given up by the count of pairs; one firm a worker: as many runs as workers
@pytest.mark.parametrize("pattern", [np.repeat([0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 0], 2), np.repeat([0, 1] * 5, 2),
                                     np.repeat(list(range(17)) * 2, 2), np.repeat([0], 6)])
@pytest.mark.parametrize("years", [0, 8])
@pytest.mark.parametrize("precision,cg", [("mixed", True), ("fp64", False)])
def test_runs_match_the_oracle(built, pattern, years, precision, cg):
    workers = 9_000 // len(pattern) * 2
    y, W, fe = panel(workers, 150, years, pattern, len(pattern) + years)
    for clusters in ([1], [2], [1, 2]):
        cfg = fe_runtime_config(fe_tolerance=1e-10, fe_max_iterations=20_000, precision=precision, demean_cg=cg,
                                cluster_fe_dims=clusters)
        got = fe_gpu_estimate(cfg, None, host(y, W, fe))
        ref = O.gpu_estimate(y, W, fe, Z=np.zeros((len(y), 0), order="F"), tol=1e-12, max_iter=200_000,
                             cluster_dims=clusters, iv_regressors=[])
        assert got.converged
        # means left at 1e-10 of unit columns
        np.testing.assert_allclose(got.beta, ref.beta, rtol=0, atol=1e-9)
        np.testing.assert_allclose(got.se, ref.se, rtol=1e-6, atol=0)


def _high(call):
    used, high, reserved = C.c_ulonglong(), C.c_ulonglong(), C.c_ulonglong()
    call()  # what the library keeps from a first call
    ref = [C.byref(used), C.byref(high), C.byref(reserved)]
    N.check(N.lib().fegb_pool_usage(1, *ref), "fegb_pool_usage")
    before = used.value
    call()
    N.check(N.lib().fegb_pool_usage(0, *ref), "fegb_pool_usage")
    return high.value - before


def test_runs_given_up_leave_no_memory_behind(built):
    """The same pairs and rows per pair, in runs of two rows (given up) and of one (not formed)"""
    cfg = fe_runtime_config(fe_tolerance=1e-6, fe_max_iterations=20, precision="mixed", demean_cg=True)
    peak = []
    for pattern in (np.repeat([0, 1] * 5, 2), np.array([0, 1] * 10)):
        y, W, fe = panel(20_000, 900, 0, pattern, 3)
        peak.append(_high(lambda: fe_gpu_within_transform(cfg, host(y, W, fe))))
    n = 20_000 * 20
    assert peak[0] <= peak[1] + n  # the pool's rounding; the arrays of the runs are 4 n and more
