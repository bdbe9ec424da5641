"""The posting-major SPFresh scan at the edges of what postings may hold,
against the oracle's restatement of the search (src/spfresh.rs:671-770)."""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import synth
from test_gpu_spfresh import oracle_view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["repeats", "gc"])
@pytest.mark.parametrize("shift", [0.0, 0.5])  # tensor-core tiles, FMA tiles (halves; sums still exact)
def test_live_postings_without_entries(oracle, how, shift):
    """Live postings whose entries have all moved away (every vector occurs
    twice: equal centroids lose their ties) or were deleted and collected.
    They are probed like any other and add nothing."""
    n = 2000 if how == "repeats" else 3000
    X = synth.mixture(n, 32, 40, seed=41, clip=False) + np.float32(shift)
    if how == "repeats":
        X = np.concatenate([X, X])
    s = dg.SPFresh.build(X, max_posting_size=16, min_posting_size=4 if how == "repeats" else 0, seed=2)
    if how == "gc":
        s.delete(np.nonzero(X[:, 0] > X[:, 0].mean())[0].tolist())
        s.gc()
    live = np.nonzero(s.live_b)[0]
    empty = [b for b in live if s._len(b) == 0]
    Q = synth.mixture(700, 32, 40, seed=41, stream=synth.STREAM_QUERY, clip=False) + np.float32(shift)
    C = np.asarray(s.cent)[live]
    D = (Q * Q).sum(1)[:, None] + (C * C).sum(1)[None] - 2.0 * Q @ C.T
    near = live[np.argsort(D, axis=1)[:, :64]]
    assert len(live) >= 512 and np.isin(near, empty).any()
    view, keep = oracle_view(oracle, s)
    for k, nprobe in ((10, 64), (1, 64), (20, 100)):
        gi, gd, gc = s.search_arrays(Q, k, nprobe)
        oi, od, oc = oracle.spfresh_search(view, Q, k, nprobe)
        assert np.array_equal(gc, oc) and np.array_equal(gi, oi) and np.array_equal(gd, od), (k, nprobe)
    s.close()
