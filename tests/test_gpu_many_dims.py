"""Within-transforms over four to eight dimensions, all of them swept (more than
64 groups) or some small: the projections take as many as a fit may have."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_within_transform, fe_runtime_config
from fe_gpu_gb300.bin_io import fe_host_arrays
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(400, 300, 200, 100), (400, 300, 200, 100, 70), (90, 80, 70, 100, 110, 9, 12),
                                   (400, 300, 200, 100, 70, 71, 72, 73), (8, 7, 6, 5, 4, 3, 2, 500)])
@pytest.mark.parametrize("order", ["random", "sorted"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_many_dimensions(built, sizes, order, precision):
    rng = np.random.default_rng(len(sizes))
    n, k = 6_000, 2
    fe = np.vstack([rng.integers(1, g + 1, size=n) for g in sizes]).astype(np.int32)
    if order == "sorted":
        fe = np.asfortranarray(fe[:, np.lexsort(fe[::-1])])
    y, W = rng.standard_normal(n), rng.standard_normal((n, k))
    host = fe_host_arrays(y=y.copy(), W=np.asfortranarray(W), Z=np.zeros((n, 0), order="F"), fe_ids=np.asfortranarray(fe))
    cfg = fe_runtime_config(fe_tolerance=1e-9, fe_max_iterations=5_000, precision=precision)
    conv, _, _ = fe_gpu_within_transform(cfg, host)
    oy, oW, _, _, oconv, _ = O.demean_symmetric(y, W, fe, 1e-11, 5_000)
    assert conv and oconv
    # means below 1e-9 in each dimension: within 20 times that of the projection for each of eight
    np.testing.assert_allclose(host.y, oy, atol=1.6e-7, rtol=0)
    np.testing.assert_allclose(host.W, oW, atol=1.6e-7, rtol=0)
