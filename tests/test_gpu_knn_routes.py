"""Exact kNN on both sides of the line between its two kernels, against the CPU oracle."""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,nq,k", [(2000, 8, 512, 40), (2000, 8, 513, 40), (2000, 16, 1024, 40),
                                      (2000, 8, 1024, 40), (2000, 8, 1025, 40), (2500, 64, 1100, 16), (2500, 64, 1100, 17),
                                      (70, 3, 1300, 70), (1, 8, 1100, 1), (90, 1025, 1030, 20)])
@pytest.mark.parametrize("metric", ["l2", "euclidean"])
def test_exact_knn_routes(oracle, n, d, nq, k, metric):
    X = synth.mixture(n, d, 4, seed=13)
    Q = synth.mixture(nq, d, 4, seed=13, stream=synth.STREAM_QUERY)
    gi, gd = dg.exact_knn(X, Q, k, metric)
    oi, od = oracle.exact_knn(X, Q, k)
    if metric == "euclidean":
        od = np.sqrt(od.astype(np.float64)).astype(np.float32)
    assert np.array_equal(gi, oi) and np.array_equal(gd, od)
