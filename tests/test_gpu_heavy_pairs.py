"""A pair of groups with more rows than FP32 counts (2^24): its weight in the
streams of the group tables has to be exact, or the demeaned rows keep means of
2^-24 of the effects."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_within_transform, fe_runtime_config
from fe_gpu_gb300.bin_io import fe_host_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["sorted", "random"])
@pytest.mark.parametrize("precision,cg", [("fp64", False), ("mixed", True)])
def test_rows_of_a_heavy_pair_are_demeaned(built, order, precision, cg):
    rng = np.random.default_rng(7)
    heavy, rest = (1 << 24) + 1, 200_000
    n = heavy + rest
    a = np.concatenate([np.zeros(heavy, np.int32), rng.integers(0, 100, rest, dtype=np.int32)])
    b = np.concatenate([np.zeros(heavy, np.int32), rng.integers(0, 90, rest, dtype=np.int32)])
    at = np.lexsort((b, a)) if order == "sorted" else rng.permutation(n)
    a, b = a[at], b[at]
    y = (30.0 * rng.standard_normal(100))[a] + (30.0 * rng.standard_normal(90))[b] + rng.standard_normal(n)
    host = fe_host_arrays(y=y, W=np.zeros((n, 0), order="F"), Z=np.zeros((n, 0), order="F"),
                          fe_ids=np.asfortranarray(np.vstack([a, b]) + 1))
    cfg = fe_runtime_config(fe_tolerance=1e-8, fe_max_iterations=20_000, precision=precision, demean_cg=cg)
    converged, _, _ = fe_gpu_within_transform(cfg, host)
    assert converged
    # the sums here: 2^24 terms below 6, rounded by 2^-53 of the running sum (below 1e5) each
    for g in (a, b):
        assert np.abs(np.bincount(g, host.y) / np.bincount(g)).max() < 1e-8 + 1e-11 * 6
