"""Alternating projections on group tables against the oracle's row-by-row
scheme, at the edges of the table forms: group counts around the 64 of a count
matrix, source tiles and their remainders, counts beyond a byte and beyond the
fixed-point range, one to four dimensions, the widest rows, empty groups and
columns with a large level (which start on the rows)."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_within_transform, fe_runtime_config
from fe_gpu_gb300.bin_io import fe_host_arrays
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ITERATIONS = 6


def panel(n, sizes, k, seed, order="random", level=0.0):
    rng = np.random.default_rng(seed)
    fe = np.vstack([rng.integers(1, g + 1, size=n) for g in sizes]).astype(np.int32)
    if order == "sorted":
        fe = fe[:, np.argsort(fe[np.argmax(sizes)], kind="stable")]
    y = rng.standard_normal(n) + level
    W = rng.standard_normal((n, k)) + 0.2 * fe[0][:, None] / sizes[0]
    return y, np.asfortranarray(W), np.asfortranarray(fe)


CASES = [
    # rows, group counts, regressors
    (900, (7,), 2),                      # one dimension: repeated projections only
    (1500, (64, 63), 1),                 # count matrices on both sides
    (3000, (65, 64), 3),                 # one more group than a count matrix holds
    (70001, (129, 3), 4),                # counts beyond a byte
    (20000, (1000, 13, 12), 5),          # counts beyond the fixed-point range, two small dimensions
    (4097, (700, 90, 9), 8),             # two swept dimensions and a small one
    (9000, (4000, 600, 20), 1),          # two columns
    (6000, (900, 40, 30, 5), 15),        # four dimensions
    (5000, (800, 64, 17), 31),           # 32 columns
    (5000, (800, 64, 17), 32),           # 33 columns: projections on the rows
    (60000, (12000, 3000, 11), 2),       # short groups and chunked groups
    (3000, (200, 9), 2),                 # one large dimension and small ones: one launch, one block
    (30000, (5000, 17, 64, 2), 8),       # the same over many blocks, pieces of 16 and their remainders
    (700, (65, 33), 31),                 # 32 columns: one slot a warp
    (3000000, (600000, 5), 3),           # more elements than the one-launch form takes
]


@pytest.mark.parametrize("n,sizes,k", CASES)
@pytest.mark.parametrize("order", ["random", "sorted"])
def test_table_projections_follow_the_rows(built, n, sizes, k, order):
    y, W, fe = panel(n, sizes, k, seed=n + k, order=order)
    host = fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((n, 0), order="F"), fe_ids=fe)
    cfg = fe_runtime_config(fe_tolerance=1e-9, fe_max_iterations=ITERATIONS)
    _, iters, mu = fe_gpu_within_transform(cfg, host)
    oy, oW, _, oit, _, omu = O.demean_symmetric(y, W, fe, 1e-9, ITERATIONS)
    assert iters == oit
    # 4 projections per dimension and iteration, each mean within 64 x 2^-53 of the
    # largest value (below 6 here): 6 x 16 x 64 x 1.1e-16 x 6 = 4e-12
    np.testing.assert_allclose(host.y, oy, atol=4e-12, rtol=0)
    np.testing.assert_allclose(host.W, oW, atol=4e-12, rtol=0)
    assert abs(mu - omu) < 4e-12


def test_large_level_starts_on_the_rows(built):
    n, sizes = 8000, (500, 30, 12)
    level = 1.0e7
    y, W, fe = panel(n, sizes, 3, seed=5, level=level)
    host = fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((n, 0), order="F"), fe_ids=fe)
    conv, iters, mu = fe_gpu_within_transform(fe_runtime_config(fe_tolerance=1e-7, fe_max_iterations=200), host)
    oy, oW, _, oit, oconv, _ = O.demean_symmetric(y, W, fe, 1e-7, 200)
    assert conv and oconv and abs(iters - oit) <= 1
    # the level's own rounding in the rows (2^-53 x 1e7 per subtraction) and one iteration's tolerance
    np.testing.assert_allclose(host.y, oy, atol=1e-6, rtol=0)
    np.testing.assert_allclose(host.W, oW, atol=1e-6, rtol=0)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n,sizes,k", [(4097, (700, 90, 9), 3), (9000, (1000, 13, 12), 3)])
def test_a_column_with_a_non_finite_value_stays_apart(built, n, sizes, k, bad):
    y, W, fe = panel(n, sizes, k, seed=3)
    ref = fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((n, 0), order="F"), fe_ids=fe)
    y[17] = bad
    host = fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((n, 0), order="F"), fe_ids=fe)
    cfg = fe_runtime_config(fe_tolerance=1e-8, fe_max_iterations=ITERATIONS)
    fe_gpu_within_transform(cfg, host)
    fe_gpu_within_transform(cfg, ref)
    assert not np.isfinite(host.y).any()  # every row is connected to row 17
    assert np.isfinite(host.W).all()
    # the relaxation goes by the largest update over all columns, so the clean
    # columns follow another path to the same limit
    assert np.abs(host.W - ref.W).max() < 1.0


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n,sizes,k", [(4097, (700, 90, 9), 3), (9000, (1000, 13, 12), 3)])
def test_clean_columns_converge_beside_a_non_finite_one(built, n, sizes, k, bad):
    y, W, fe = panel(n, sizes, k, seed=3)
    out = []
    for first in (y[17], bad):
        y[17] = first
        host = fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((n, 0), order="F"), fe_ids=fe)
        conv, iters, _ = fe_gpu_within_transform(fe_runtime_config(fe_tolerance=1e-10, fe_max_iterations=500), host)
        assert conv and iters < 200
        out.append(host.W)
    # updates below 1e-10 at a rate of at most 0.9 an iteration (these panels converge in a few dozen) leave 1e-9 each
    np.testing.assert_allclose(out[1], out[0], atol=2e-9, rtol=0)


@pytest.mark.parametrize("n,sizes,k", [c for c in CASES if len(c[1]) > 1 and c[0] < 1_000_000])
@pytest.mark.parametrize("order", ["random", "sorted"])
def test_mixed_form_reaches_the_fp64_limit(built, n, sizes, k, order):
    y, W, fe = panel(n, sizes, k, seed=n + k, order=order)
    out = []
    for precision, tol in (("mixed", 1e-9), ("fp64", 1e-11)):
        host = fe_host_arrays(y=y.copy(), W=W.copy(order="F"), Z=np.zeros((n, 0), order="F"), fe_ids=fe)
        cfg = fe_runtime_config(fe_tolerance=tol, fe_max_iterations=2000, precision=precision)
        conv, _, _ = fe_gpu_within_transform(cfg, host)
        assert conv
        out.append(np.column_stack([host.y, host.W]))
    # means below 1e-9 in every dimension; the projection on these panels' dimensions (a few dozen iterations)
    # is at most 20 times the largest mean of each of up to four
    np.testing.assert_allclose(out[0], out[1], atol=8e-8, rtol=0)
