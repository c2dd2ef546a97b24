"""Which dimensions are held as count matrices: their bound counts the padding of
the rows that the group tables read (16 counts and multiples of it)."""
import ctypes as C

import pytest

from fe_gpu_gb300 import _native as N


def plan(sizes, columns, padded):
    out = (C.c_int * len(sizes))()
    N.check(N.lib().fegb_test_dense_plan((C.c_int * len(sizes))(*sizes), len(sizes), columns, 10**9, padded, out),
            "fegb_test_dense_plan")
    return list(out)


# 8e9 bytes at 4 a count: 1e9 groups of 2 counts, or 125e6 of 16 with the padding
@pytest.mark.parametrize("sizes,columns,padded,want", [
    ((1000, 13, 12), 4, 0, [0, 1, 1]), ((1000, 13, 12), 4, 1, [0, 1, 1]), ((1000, 65), 4, 1, [0, 0]),
    ((1000, 64), 33, 1, [0, 0]), ((1000, 64), 32, 1, [0, 1]),
    ((124_000_000, 2), 4, 1, [0, 1]), ((126_000_000, 2), 4, 1, [0, 0]), ((126_000_000, 2), 4, 0, [0, 1]),
    ((999_000_000, 2), 4, 0, [0, 1]), ((1_000_000_001, 2), 4, 0, [0, 0]),
    ((62_000_000, 30), 4, 1, [0, 1]), ((63_000_000, 30), 4, 1, [0, 0]), ((66_000_000, 30), 4, 0, [0, 1])])
def test_bound_counts_the_padding(built, sizes, columns, padded, want):
    assert plan(sizes, columns, padded) == want
