"""Mixed projections at their iteration limit: an inner solve takes at most half of
the iterations that are left and the refinement goes on from FP64 means, so a
limit of m iterations is the FP64 form in pieces of ceil(m / 2), ... iterations,
each from the start of its relaxation."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_within_transform, fe_runtime_config
from fe_gpu_gb300.bin_io import fe_host_arrays

pytestmark = pytest.mark.gpu


def pieces(limit):
    while limit > 0:
        yield (limit + 1) // 2
        limit -= (limit + 1) // 2


@pytest.mark.parametrize("sizes,k", [((4,), 2), ((900,), 2), ((50, 20), 3), ((3000, 700, 9), 2), ((40, 30), 33)])
@pytest.mark.parametrize("limit", [1, 2, 3, 5, 8])
def test_limit_is_spent_in_halves(built, sizes, k, limit):
    rng = np.random.default_rng(1)
    n = 20_000 if max(sizes) > 100 else 400
    fe = np.asfortranarray(np.vstack([rng.integers(1, g + 1, size=n) for g in sizes]).astype(np.int32))
    y, W = rng.standard_normal(n), np.asfortranarray(rng.standard_normal((n, k)))

    def host(y, W):
        return fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((n, 0), order="F"), fe_ids=fe)

    got = host(y, W)
    conv, iters, _ = fe_gpu_within_transform(
        fe_runtime_config(fe_tolerance=1e-13, fe_max_iterations=limit, precision="mixed"), got)
    assert iters == limit
    want = host(y, W)
    for m in pieces(limit):
        fe_gpu_within_transform(fe_runtime_config(fe_tolerance=1e-13, fe_max_iterations=m), want)
    # FP32 projections: 2^-24 of values below 6, some 50 roundings deep
    np.testing.assert_allclose(got.y, want.y, atol=2e-5, rtol=0)
    np.testing.assert_allclose(got.W, want.W, atol=2e-5, rtol=0)
