"""The CTA-per-query beam search at every CTA width, against the CPU oracle.

The width follows from the number of queries (8, 4, 2 and 1 warps per query as
the batch grows), so the batch sizes here sit on both sides of each boundary
of a 148-SM GPU.  Integer-valued data: every distance is exact, so ids, counts
and distances must equal the oracle's bit for bit.
"""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import _lib, synth

pytestmark = pytest.mark.gpu

N, D = 1500, 40  # a row of 64 padded floats; 16-candidate tiles and list words end raggedly


def _index(degree, seed, repeats):
    """A random graph (degree not a multiple of 4 or of the warps); with repeats, rows
    list some neighbours twice and end in padding."""
    X = synth.mixture(N, D, 16, seed=seed)
    rng = np.random.default_rng(seed)
    adj = rng.integers(0, N, (N, degree)).astype(np.uint32)
    if repeats:
        adj[:, 1::3] = adj[:, :1]
        adj[::2, -1] = _lib.PAD
    return X, adj


@pytest.fixture(scope="module", params=[(13, False), (70, True), (64, False)], ids=["r13", "r70rep", "r64"])
def pair(request, oracle):
    degree, repeats = request.param
    X, adj = _index(degree, degree, repeats)
    labels = (np.arange(N, dtype=np.uint64)[:, None] * np.array([1, 7], dtype=np.uint64)) % np.uint64(5)
    g = dg.FilteredDiskANN(X, adj, 3, labels)
    g.enable_bf16()
    o = oracle.OracleIndex(X, adj, 3)
    o.set_labels(labels)
    yield g, o
    g.close()


def _same(g, o):
    for a, b in zip((g[2], g[0], g[1]), (o[2], o[0], o[1])):
        assert np.array_equal(np.asarray(a), b)


@pytest.mark.parametrize("nq", [1, 297, 741, 1481])
@pytest.mark.parametrize("L,k", [(5, 3), (65, 10), (257, 10), (1000, 1000)])
def test_widths(pair, nq, L, k):
    g, o = pair
    if L == 1000 and nq > 300:
        nq = nq // 4
    Q = synth.mixture(nq, D, 16, seed=5, stream=synth.STREAM_QUERY)
    _same(g.search_arrays(Q, k, L), o.search(Q, k, L))
    r = min(L, 1024)
    _same(g.search_arrays(Q, k, L, traversal=_lib.TRAVERSE_BF16, rerank_size=r), o.search(Q, k, L))


@pytest.mark.parametrize("nq", [1, 297, 1481])
@pytest.mark.parametrize("L,k", [(3, 1), (40, 10), (20, 100)])
def test_widths_filtered(pair, nq, L, k):
    g, o = pair
    Q = synth.mixture(nq, D, 16, seed=6, stream=synth.STREAM_QUERY)
    f = dg.Filter.or_([dg.Filter.eq(0, 2), dg.Filter.and_([dg.Filter.gt(1, 2), dg.Filter.lt(0, 2)])])
    ops, pool = f.program()
    _same(g.search_arrays(Q, k, L, filters=f), o.search(Q, k, L, filter_ops=ops, filter_pool=pool))
