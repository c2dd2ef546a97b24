"""The bounded wait of the projections in one launch: a limit of zero makes every
block give up at the first barrier that is not complete; the call reports it and
the next one, with the usual limit, gives its results again. (Nothing hangs: each
block leaves by itself.) Repeated calls give the same bits."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_within_transform, fe_runtime_config
from fe_gpu_gb300 import _native as N
from fe_gpu_gb300.bin_io import fe_host_arrays

pytestmark = pytest.mark.gpu


def transform():
    rng = np.random.default_rng(11)
    n = 60_000
    fe = np.vstack([rng.integers(1, g + 1, size=n) for g in (20_000, 17, 12)]).astype(np.int32)
    y, W = rng.standard_normal(n), rng.standard_normal((n, 5))
    host = fe_host_arrays(y=y, W=np.asfortranarray(W), Z=np.zeros((n, 0), order="F"), fe_ids=np.asfortranarray(fe))
    fe_gpu_within_transform(fe_runtime_config(fe_tolerance=1e-8, fe_max_iterations=500), host)
    return host


def test_a_wait_that_runs_out_is_an_error_and_the_next_call_works(built):
    want = transform()
    try:
        N.check(N.lib().fegb_test_projection_wait(0), "fegb_test_projection_wait")
        with pytest.raises(N.FeGpuError, match="ran out of time"):
            transform()
    finally:
        N.check(N.lib().fegb_test_projection_wait(-1), "fegb_test_projection_wait")
    for _ in range(3):
        again = transform()
        np.testing.assert_array_equal(again.y, want.y)
        np.testing.assert_array_equal(again.W, want.W)
