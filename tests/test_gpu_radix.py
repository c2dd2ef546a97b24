"""Radix sorts and scans behind the integer preparation at tile and digit
edges: cluster ids (a 32- or 64-bit key sort by the key span) against numpy's
ranks."""
import ctypes as C

import numpy as np
import pytest

from fe_gpu_gb300 import DeviceBuffer
from fe_gpu_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 4095, 4096, 4097, 8191, 8192, 8193, 70001])
@pytest.mark.parametrize("sizes", [(2,), (255,), (512,), (513,), (5000, 90), (100000, 3000), (2000000, 70000, 30)])
def test_cluster_ids_are_key_ranks(built, n, sizes):
    rng = np.random.default_rng(n + sum(sizes))
    ids = [rng.integers(1, g + 1, size=n).astype(np.int32) for g in sizes]
    for v, g in zip(ids, sizes):
        v[-1] = g  # the largest key of the span
    key = np.zeros(n, dtype=np.uint64)
    stride = np.uint64(1)
    for v, g in zip(ids, sizes):
        key += (v.astype(np.uint64) - np.uint64(1)) * stride
        stride *= np.uint64(g)
    _, want = np.unique(key, return_inverse=True)
    bufs = [DeviceBuffer.from_array(v) for v in ids]
    out = DeviceBuffer(4 * n)
    ptrs = (C.c_void_p * len(bufs))(*[C.c_void_p(b.ptr) for b in bufs])
    cnt = C.c_int(0)
    N.check(N.lib().fegb_cluster_ids(ptrs, N.int_array(list(sizes)), len(sizes), n, C.c_void_p(out.ptr), C.byref(cnt)),
            "fegb_cluster_ids")
    got = out.to_array(np.int32, (n,))
    assert cnt.value == want.max() + 1
    np.testing.assert_array_equal(got, want.reshape(-1) + 1)
