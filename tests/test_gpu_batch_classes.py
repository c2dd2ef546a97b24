"""Column classes of a batch side by side on threads and streams: the same bits
as one class at a time (profiled fits), call after call, with more classes than
threads; an error in one class is the call's error and leaves the next call
whole."""
import numpy as np
import pytest

from fe_gpu_gb300 import _native as N
from fe_gpu_gb300.estimator import DeviceBuffer, fe_batch_spec, fe_gpu_estimate_batch, fe_runtime_config

pytestmark = pytest.mark.gpu

COLUMNS = (2, 6, 10, 14, 20, 28, 40, 55)  # eight classes: 4, 8, 12, 16, 24, 32, 48, 64 columns


def upload(bad=None):
    keep, rows = [], []
    for s in range(3 * len(COLUMNS)):
        r = np.random.RandomState(s)
        k, n = COLUMNS[s % len(COLUMNS)], int(np.exp(r.uniform(np.log(1_000), np.log(40_000))))
        sizes = [max(2, int(0.4 * n ** 0.7)), 9, 40][:1 + s % 3]
        ids = [r.randint(1, m + 1, n).astype(np.int32) for m in sizes]
        W = r.normal(size=(k, n))
        y = W.sum(0) + r.normal(size=n) + (0.3 * r.normal(size=sizes[0] + 1))[ids[0]]
        if s == bad:
            ids[0][n // 2] = 0
        b = [DeviceBuffer.from_array(v) for v in [y, W] + ids]
        keep.append(b)
        rows.append(fe_batch_spec(n=n, k=k, l=0, d_y=b[0].ptr, d_W=b[1].ptr, d_Z=None, d_fe_ids=[v.ptr for v in b[2:]],
                                  cluster_fe_dims=list(range(1, 1 + s % (len(sizes) + 1))), iv_regressors=[]))
    return keep, rows


def fit(rows, profile=False):
    res = fe_gpu_estimate_batch(fe_runtime_config(fe_tolerance=1e-8, fe_max_iterations=20_000, precision="mixed",
                                                  demean_cg=True), rows, profile=profile)
    return [np.concatenate([r.beta, r.se, [r.rss, r.tss_within, r.fe_iterations, r.converged]]) for r in res]


def test_classes_side_by_side_give_the_bits_of_one_at_a_time(built):
    keep, rows = upload()
    want = fit(rows, profile=True)
    for _ in range(4):
        for a, b in zip(fit(rows), want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("bad", [0, 7, 12])
def test_an_error_in_one_class_is_reported(built, bad):
    keep, rows = upload(bad)
    with pytest.raises(N.FeGpuError, match=f"spec {bad}: FE dimension 1 has an id < 1"):
        fit(rows)
    keep, rows = upload()
    for a, b in zip(fit(rows), fit(rows, profile=True)):
        np.testing.assert_array_equal(a, b)
