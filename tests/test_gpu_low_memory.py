"""Device memory that runs out in the middle of a call (failed allocations, no
memory used up): a fit without room for the group tables goes on with its rows, a
batch class without room beside others runs alone afterwards, and what cannot be
done is an error that leaves the next call whole."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_estimate, fe_runtime_config
from fe_gpu_gb300 import _native as N
from fe_gpu_gb300.bin_io import fe_host_arrays
from tests.test_gpu_batch_classes import fit, upload

pytestmark = pytest.mark.gpu


@pytest.fixture
def failing():
    yield lambda what, times: N.check(N.lib().fegb_test_fail_alloc(what, times), "fegb_test_fail_alloc")
    N.check(N.lib().fegb_test_fail_alloc(None, 0), "fegb_test_fail_alloc")


def panel(runs):
    rng = np.random.default_rng(5)
    n = 30_000
    w = np.repeat(np.arange(n // 10), 10)
    f = rng.integers(0, 200, (n // 10, 2))[w, np.tile(np.repeat([0, 1], 5) if runs else np.arange(10) % 2, n // 10)]
    t = np.tile(np.arange(10), n // 10)
    at = np.arange(n) if runs else rng.permutation(n)
    W = rng.standard_normal((n, 4)) + 0.2 * rng.standard_normal(200)[f][:, None]
    y = W.sum(1) + rng.standard_normal(200)[f] + rng.standard_normal(n // 10)[w] + rng.standard_normal(n)
    fe = np.vstack([w, f, t]).astype(np.int32)[:, at] + 1
    return y[at], np.asfortranarray(W[at]), np.asfortranarray(fe)


TABLES = [b"group tables", b"small-dimension counter", b"increments taken out"]
STREAMS = [b"combined increments", b"tuple group offsets", b"count matrix (uint8)"]  # a CG operator needs its own


@pytest.mark.parametrize("what,precision,cg", [(w, p, False) for p in ("fp64", "mixed") for w in TABLES + STREAMS]
                         + [(w, p, True) for p in ("fp64", "mixed") for w in TABLES])
@pytest.mark.parametrize("runs", [True, False])
def test_a_fit_without_room_for_tables_runs_on_its_rows(built, failing, what, precision, cg, runs):
    y, W, fe = panel(runs)
    cfg = fe_runtime_config(fe_tolerance=1e-10, fe_max_iterations=5_000, precision=precision, demean_cg=cg,
                            cluster_fe_dims=[1, 2])

    def run():
        host = fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((len(y), 0), order="F"), fe_ids=fe)
        return fe_gpu_estimate(cfg, None, host)

    want = run()
    failing(what, 1)
    got = run()
    assert got.converged and want.converged
    # both below means of 1e-10 of unit columns
    np.testing.assert_allclose(got.beta, want.beta, rtol=0, atol=1e-9)
    np.testing.assert_allclose(got.se, want.se, rtol=1e-7, atol=0)


def test_batch_classes_without_room_run_alone(built, failing):
    keep, rows = upload()
    want = fit(rows)
    failing(b"stacked y", 3)
    for a, b in zip(fit(rows), want):
        np.testing.assert_array_equal(a, b)
    failing(b"stacked y", 1000)
    with pytest.raises(N.FeGpuError, match="stacked y: out of memory"):
        fit(rows)
    failing(None, 0)
    for a, b in zip(fit(rows), want):
        np.testing.assert_array_equal(a, b)
