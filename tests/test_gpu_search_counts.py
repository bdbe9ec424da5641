"""The counts of a search (expanded and evaluated ids) do not depend on how
many queries share its call, for states so large that few queries fit an SM."""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quant,L", [("pq", 128), ("int8cos", 200)])
def test_counts_at_any_batch_size(quant, L):
    """PQ tables of 16 KB and 768-d cosine codes: the beam's visited table
    forgets ids, so a smaller one would show in the counts."""
    rng = np.random.default_rng(3)
    n, nq = 20_000, 1_500  # above five queries per SM
    if quant == "pq":
        X = synth.mixture(n, 32, 16, seed=3)
        Q = synth.mixture(nq, 32, 16, seed=3, stream=synth.STREAM_QUERY)
    else:
        X, Q = synth.cosine(n, nq, 768, seed=3)
    adj = rng.integers(0, n, (n, 48)).astype(np.uint32)
    g = dg.QuantizedDiskANN(X, adj, 0, "l2" if quant == "pq" else "cosine", rerank_size=64)
    if quant == "pq":
        g.attach_pq(dg.pq_train(X[:4096], 16, 256, 2, 4096, seed=1))
    else:
        g.attach_int8(*dg.int8_params(X))
    kw = dict(traversal=_lib.TRAVERSE_CODES, rerank_size=64)
    ids, ds, cnt, st = g.search_arrays(Q, 10, L, with_stats=True, **kw)
    for s in range(0, nq, 300):
        i, d, c, t = g.search_arrays(Q[s:s + 300], 10, L, with_stats=True, **kw)
        assert np.array_equal(t, st[s:s + 300])
        assert np.array_equal(i, ids[s:s + 300]) and np.array_equal(d, ds[s:s + 300]) and np.array_equal(c, cnt[s:s + 300])
    i, d, c = g.search_arrays(Q, 10, L, **kw)  # without the counts: another table, the same results
    assert np.array_equal(i, ids) and np.array_equal(d, ds) and np.array_equal(c, cnt)
    g.close()
