"""Within-transforms whose increments are far larger than the group means: means
predicted from group tables are uncertain by some 2^-53 of the increments, and
"converged" speaks of the rows' own means."""
import numpy as np
import pytest

from fe_gpu_gb300 import fe_gpu_within_transform, fe_runtime_config
from fe_gpu_gb300.bin_io import fe_host_arrays

pytestmark = pytest.mark.gpu

TOL = 1e-8


def two_clusters(n, shift):
    """Two sets of n persons with a row at their set's large firm and one at one of its 40 small firms, linked by one
    person with a row of -shift / 2 in the one and shift / 2 in the other: means of shift / (2 n), increments of
    shift / 2"""
    rng = np.random.default_rng(n)
    person, firm = [], []
    for c in (0, 1):
        p = c * n + np.arange(n)
        person += [p, p]
        firm += [np.full(n, 41 * c), 41 * c + 1 + rng.integers(0, 40, n)]
    person = np.concatenate(person + [np.array([2 * n, 2 * n])])
    firm = np.concatenate(firm + [np.array([0, 41])])
    y = rng.standard_normal(len(person))
    y[-2:] = -0.5 * shift, 0.5 * shift
    return y, rng.standard_normal((len(y), 1)), np.asfortranarray(np.vstack([person, firm]).astype(np.int32) + 1)


def chain(links, size, copies):
    """y = a + b, b = size cos(pi i / links) along a chain of nodes and a minus its mean in each of the links, which come
    copies times over: group means of size (pi / links)^2 / 4 at most"""
    rng = np.random.default_rng(links)
    link = np.repeat(np.arange(links * copies), 2)
    step = link % links
    node = step + np.tile([0, 1], links * copies)
    b = size * np.cos(np.pi * np.arange(links + 1) / links)
    y = b[node] - 0.5 * (b[step] + b[step + 1])
    return y, rng.standard_normal((len(y), 2)), np.asfortranarray(np.vstack([link, node]).astype(np.int32) + 1)


def largest_mean(columns, ids):
    out = 0.0
    for i in ids:
        n = np.maximum(np.bincount(i - 1), 1)
        for c in columns:
            out = max(out, np.abs(np.bincount(i - 1, c) / n).max())
    return out


def transform(y, W, fe, **cfg):
    host = fe_host_arrays(y=y.copy(), W=np.asfortranarray(W), Z=np.zeros((len(y), 0), order="F"), fe_ids=fe)
    converged, iterations, _ = fe_gpu_within_transform(fe_runtime_config(fe_tolerance=TOL, **cfg), host)
    return converged, iterations, host


@pytest.mark.parametrize("precision,n", [("mixed", 1_000), ("fp64", 4_000), ("fp64", 100_000), ("fp64", 400_000)])
def test_converged_holds_on_the_rows(built, precision, n):
    y, W, fe = two_clusters(n, 2.0 * n * 1200.0)  # means of 1200: below the tables' limit of 1400 at this tolerance
    converged, _, host = transform(y, W, fe, fe_max_iterations=20_000, precision=precision, demean_cg=True)
    assert converged
    # the means of the returned columns (below 10), themselves rounded by 2^-53 of 400,000 terms at most
    assert largest_mean([host.y, host.W[:, 0]], fe) < TOL + 5e-10


# 41 / 70 links: two small dimensions / two large ones; 30 links ten times: one large and one small (one launch)
@pytest.mark.parametrize("links,copies", [(41, 1), (70, 1), (30, 10)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_projections_beyond_the_tables_limit(built, precision, links, copies):
    size = 600.0 * 4.0 * (links / np.pi) ** 2  # means of 600, increments of 2e5 and more
    y, W, fe = chain(links, size, copies)
    converged, _, host = transform(y, W, fe, fe_max_iterations=200_000, precision=precision)
    assert converged
    assert largest_mean([host.y, *host.W.T], fe) < TOL + 1e-14
    # y lies in the span of the dimensions: means below TOL leave at most TOL (links / pi)^2 of it, twice over
    assert np.abs(host.y).max() < 8.0 * TOL * (links / np.pi) ** 2
