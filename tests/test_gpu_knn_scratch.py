"""Device memory that an exact kNN call takes beside its rows and results."""
import ctypes

import numpy as np
import pytest

import pydiskann_b200 as dg

pytestmark = pytest.mark.gpu

USED_MEM_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH


def test_partial_lists_stay_bounded():
    """50k queries, k = 128: one slice's lists take 51 MB.  The slices are as
    many as a quarter of a gigabyte holds, not as many as balance best."""
    n, nq, k = 1_000_000, 50_000, 128
    rng = np.random.default_rng(0)
    X, Q = np.zeros((n, 32), np.float32), np.zeros((nq, 32), np.float32)  # one coordinate that differs
    X[:, 0], Q[:, 0] = rng.integers(0, 1 << 22, n), rng.integers(0, 1 << 22, nq)
    dg.exact_knn(X[:100], Q[:2], 1)  # the context and the pool exist
    cu = ctypes.CDLL("libcuda.so.1")
    pool, dev = ctypes.c_void_p(), ctypes.c_int()
    assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), dev) == 0
    high = ctypes.c_uint64(0)
    assert cu.cuMemPoolSetAttribute(pool, USED_MEM_HIGH, ctypes.byref(high)) == 0
    ids, ds = dg.exact_knn(X, Q, k)
    assert cu.cuMemPoolGetAttribute(pool, USED_MEM_HIGH, ctypes.byref(high)) == 0
    rows, staging, results = (n + nq) * 32 * 4, 16 << 20, nq * k * 8
    assert rows + results < high.value <= rows + staging + results + (256 << 20) + (8 << 20)
    for q in (0, 777, nq - 1):
        D = (X[:, 0] - Q[q, 0]).astype(np.float64) ** 2
        want = np.lexsort((np.arange(n), D.astype(np.float32)))[:k]
        assert np.array_equal(ids[q], want) and np.array_equal(ds[q], D[want].astype(np.float32))
