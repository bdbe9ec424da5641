"""Exact kNN and PQ kernels at the edges of their tiles, against the CPU oracle.

Integer-valued data: distances, running sums and cluster sums are exact in any
order, so ids, codes and codebooks must equal the oracle's bit for bit.
"""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,nq,k", [(1, 1, 1, 1), (63, 33, 64, 5), (65, 16, 65, 16), (700, 100, 3, 128),
                                      (700, 20, 70, 129), (5000, 48, 200, 17)])
@pytest.mark.parametrize("metric", ["l2", "euclidean"])
def test_exact_knn_edges(oracle, n, d, nq, k, metric):
    X = synth.mixture(n, d, 4, seed=3)
    Q = synth.mixture(nq, d, 4, seed=3, stream=synth.STREAM_QUERY)
    gi, gd = dg.exact_knn(X, Q, k, metric)
    oi, od = oracle.exact_knn(X, Q, k)
    if metric == "euclidean":
        od = np.sqrt(od.astype(np.float64)).astype(np.float32)
    assert np.array_equal(gi, oi) and np.array_equal(gd, od)


def test_exact_knn_cosine_against_float64():
    X = np.random.default_rng(0).standard_normal((3000, 72)).astype(np.float32)
    Q = np.random.default_rng(1).standard_normal((90, 72)).astype(np.float32)
    _, gd = dg.exact_knn(X, Q, 10, "cosine")
    Xd, Qd = X.astype(np.float64), Q.astype(np.float64)
    D = 1.0 - Qd @ Xd.T / (np.linalg.norm(Qd, axis=1)[:, None] * np.linalg.norm(Xd, axis=1)[None])
    # the FP64 value rounded to FP32, and the FP64 sums' own rounding of up to 72 terms
    assert np.abs(gd - np.sort(D, axis=1)[:, :10]).max() <= 2.0 ** -24 + 72 * 2.0 ** -50


@pytest.mark.parametrize("ds", [1, 2, 3, 4, 6, 8, 10, 12, 16, 20])
@pytest.mark.parametrize("K", [1, 7, 256])
def test_pq_encode_widths(oracle, ds, K):
    M = 3
    X = synth.mixture(1500, M * ds, 8, seed=4)
    cb = synth.mixture(M * K, ds, 8, seed=5).reshape(M, K, ds)
    assert np.array_equal(dg.pq_encode(X, cb), oracle.pq_encode(X, cb))


@pytest.mark.parametrize("ds", [2, 4, 6, 8, 10, 12, 16])
def test_pq_encode_near_ties(oracle, ds):
    """Rows halfway between two centroids of inexact values: which one is nearer is decided by the
    rounding of every product and sum, so a contracted one shows."""
    M, K, n = 2, 64, 30_000
    rng = np.random.default_rng(ds)
    cb = (rng.standard_normal((M, K, ds)) * 50).astype(np.float32)
    a, b = rng.integers(0, K, (2, n, M))
    m = np.arange(M)
    X = ((cb[m, a] + cb[m, b]) * np.float32(0.5)).reshape(n, M * ds)
    assert np.array_equal(dg.pq_encode(X, cb), oracle.pq_encode(X, cb))


@pytest.mark.parametrize("n,ds,K", [(40, 4, 64), (1025, 8, 32), (5000, 3, 256), (2600, 40, 16)])
def test_pq_train_blocks(oracle, n, ds, K):
    X = synth.mixture(n, 2 * ds, 8, seed=6)
    got = dg.pq_train(X, 2, K, 4, 50_000, seed=9)
    assert np.array_equal(got, oracle.pq_train(X, 2, K, 4, 50_000, seed=9))


@pytest.mark.parametrize("d,centres,sigma,R,Lb", [(33, 4, 20.0, 5, 20), (128, 8, 20.0, 64, 128), (16, 1, 1.0, 24, 40),
                                                  (257, 4, 20.0, 16, 30), (40, 8, 20.0, 16, 200)])
@pytest.mark.parametrize("shift", [0.0, 0.5])
def test_vamana_prune_batches(oracle, d, centres, sigma, R, Lb, shift):
    """Tensor-core batches (integers whose sums stay below 2^24), FMA batches (halves: not
    integers, but every sum still exact; 257-d: sums past the bound), pools of repeats (sigma 1)
    and pools above 512 entries (beam 200): the oracle's graph, edge for edge."""
    X = synth.mixture(900, d, centres, seed=8, sigma=sigma) + np.float32(shift)
    adj, med = dg.build_graph(X, R, Lb, 1.2, seed=5)
    want, _ = oracle.build_vamana(X, R, Lb, 1.2, seed=5, medoid_id=med)
    assert np.array_equal(adj, want)


@pytest.mark.parametrize("n,d", [(11_000, 100), (40_000, 33), (9_000, 128)])
def test_staged_upload(n, d):
    """Uploads of several pinned pieces, rows padded on the device or not, from two threads at
    once (one of them takes the plain copy): the rows come back as their own nearest neighbours."""
    import threading

    X = np.random.default_rng(n).permutation(n * d).reshape(n, d).astype(np.float32)
    pick = np.linspace(0, n - 1, 50).astype(int)
    out = [None, None]

    def work(i):
        out[i] = dg.exact_knn(X, X[pick], 1)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for ids, ds in out:
        assert np.array_equal(ids[:, 0], pick) and not ds.any()
