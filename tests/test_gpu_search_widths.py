"""A query's results are the same bits at every batch size.

The batch size chooses the kernel (one warp per query with the list in
registers, or a CTA of 8, 4, 2 or 1 warps) and with it the routine that takes
the distances (tiles of 8, 16 or 32 candidates).  Real-valued data, so that
another order of summation would show; the smallest batch is what the tests
against the oracle run.  Base + delta searches are checked against the oracle
at each width.
"""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import _lib
from test_gpu_incremental import _check

pytestmark = pytest.mark.gpu

N, NQ = 3000, 1481  # 148 SMs: 8 warps up to 296 queries, 4 up to 740, 2 up to 1480, 1 above
SIZES = (1, 296, 297, 740, 741, 1480)


def _data(d, metric):
    rng = np.random.default_rng(d)
    C = rng.standard_normal((16, d)) * 2.0
    X = (C[rng.integers(0, 16, N)] + rng.standard_normal((N, d))).astype(np.float32)
    Q = (C[rng.integers(0, 16, NQ)] + rng.standard_normal((NQ, d))).astype(np.float32)
    if metric == "cosine":
        X /= np.linalg.norm(X, axis=1, keepdims=True)
        Q /= np.linalg.norm(Q, axis=1, keepdims=True)
    adj = rng.integers(0, N, (N, 37)).astype(np.uint32)
    return X, np.ascontiguousarray(Q), adj


def _index(trav, X, adj, metric):
    if trav in ("f32", "bf16", "fp8"):
        ix = dg.FilteredDiskANN(X, adj, 3, np.arange(N, dtype=np.uint64)[:, None] % np.uint64(7), metric)
        if trav == "bf16":
            ix.enable_bf16()
        elif trav == "fp8":
            ix.enable_fp8()
        return ix, {"f32": _lib.TRAVERSE_F32, "bf16": _lib.TRAVERSE_BF16, "fp8": _lib.TRAVERSE_FP8}[trav]
    ix = dg.QuantizedDiskANN(X, adj, 3, metric)
    if trav == "pq":  # M is not a multiple of 16
        ix.attach_pq(dg.pq_train(X, 10 if X.shape[1] % 10 == 0 else 24, 64, 2, N, seed=1))
    elif trav == "int8":
        ix.attach_int8(*dg.int8_params(X))
    elif trav == "f16":
        ix.attach_f16()
    else:
        ix.attach_rabitq(*dg.rabitq_params(X, 0))
    return ix, _lib.TRAVERSE_CODES


def _agree(ix, Q, k, L, **kw):
    per = {n: kw.pop(n) for n in ("per_query_beam", "per_query_k") if n in kw}
    want = ix.search_arrays(Q, k, L, **per, **kw)
    for m in SIZES:
        got = ix.search_arrays(Q[:m], k, L, **{n: v[:m] for n, v in per.items()}, **kw)
        for g, w in zip(got, want):
            assert np.array_equal(g, w[:m]), (m, L, kw)


@pytest.mark.parametrize("trav", ["f32", "bf16", "fp8", "pq", "int8", "f16", "rabitq"])
@pytest.mark.parametrize("d,metric", [(100, "l2"), (100, "euclidean"), (768, "cosine"), (100, "dot")])
def test_batch_sizes_agree(trav, d, metric):
    X, Q, adj = _data(d, metric)
    ix, t = _index(trav, X, adj, metric)
    for L, rr in ((40, 0), (40, 40), (70, 0), (150, 40)):
        _agree(ix, Q, 10, L, traversal=t, rerank_size=rr)
    rng = np.random.default_rng(1)
    _agree(ix, Q, 10, 64, traversal=t, rerank_size=20, per_query_beam=rng.integers(1, 200, NQ).astype(np.uint32),
           per_query_k=rng.integers(1, 11, NQ).astype(np.uint32))
    ix.close()


@pytest.mark.parametrize("trav", ["f32", "bf16", "fp8"])
@pytest.mark.parametrize("d,metric", [(100, "l2"), (768, "cosine")])
def test_filtered_batch_sizes_agree(trav, d, metric):
    X, Q, adj = _data(d, metric)
    ix, t = _index(trav, X, adj, metric)
    f = dg.Filter.or_([dg.Filter.eq(0, 2), dg.Filter.gt(0, 5)])
    for k, L, rr in ((1, 3, 0), (10, 40, 40), (60, 40, 0)):
        _agree(ix, Q, k, L, traversal=t, rerank_size=rr, filters=f)
    ix.close()


@pytest.mark.parametrize("nq", [1, 297, 741, 1481])
@pytest.mark.parametrize("deleted", [False, True])
def test_base_and_delta_at_each_width(oracle, small_data, nq, deleted):
    """Two seeds, and tombstones: against the oracle."""
    X, Q = small_data
    badj, bmed = oracle.build_vamana(X[:3000], R=32, L_build=64, alpha=1.2, seed=3)
    ix = dg.IncrementalDiskANN(X[:3000], badj, bmed)
    ix.add_vectors(X[3000:3200])
    if deleted:
        ix.delete_vectors(list(range(0, 3000, 9)))
    Qn = np.concatenate([Q] * (nq // len(Q) + 1))[:nq]
    for k, L in ((10, 40), (10, 100), (3, 1)):
        _check(ix, oracle, np.ascontiguousarray(Qn), k, L)
    ix.close()
