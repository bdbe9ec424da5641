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


def _norm_order(X):
    """|x|^2 as the scan sums it: four chains of FMAs over every fourth
    coordinate, then (0 + 1) + (2 + 3).  The products are whole numbers below
    2^53, so rounding an FP64 sum once is the FMA."""
    s = np.zeros((len(X), 4), dtype=np.float32)
    for i in range(0, X.shape[1], 4):
        x = X[:, i:i + 4].astype(np.float64)
        s = (x * x + s.astype(np.float64)).astype(np.float32)
    return (s[:, 0] + s[:, 1]) + (s[:, 2] + s[:, 3])


@pytest.mark.parametrize("d", [16, 96])
@pytest.mark.parametrize("company", [False, True])
def test_entry_norms_past_exact_sums(d, company):
    """Rows whose |x|^2 exceeds 2^24 rounds, so its order of summation shows.
    Small queries keep q.x exact (tensor-core tiles); large ones beside them
    in the batch send the same tiles to the FMA chain.  Either way the small
    queries' distances are |q|^2 + |x|^2 - 2 q.x in the one order."""
    X = synth.mixture(6000, d, 40, seed=43, sigma=30.0) * np.float32(8.0)
    X += np.random.default_rng(1).integers(0, 8, X.shape)  # odd ones among them: a sum of multiples of 8 is exact
    assert X.max() <= 2048.0 and (_norm_order(X) != (X.astype(np.float64) ** 2).sum(1)).mean() > 0.2
    s = dg.SPFresh.bulk_load(X, max_posting_size=20, seed=3)
    live = int(np.sum(s.live_b))
    assert 512 <= live <= 1024
    small = np.random.default_rng(0).integers(0, 80, (600, d)).astype(np.float32)
    Q = np.concatenate([small, X[:600]]).reshape(2, 600, d).swapaxes(0, 1).reshape(1200, d) if company else small
    gi, gd, gc = s.search_arrays(np.ascontiguousarray(Q), 20, 1024)
    if company:
        gi, gd, gc = gi[::2], gd[::2], gc[::2]
    qn = (small.astype(np.float64) ** 2).sum(1).astype(np.float32)  # exact, as every q.x
    dot = (small.astype(np.float64) @ X.T.astype(np.float64)).astype(np.float32)
    D = np.maximum((qn[:, None] + _norm_order(X)[None]) - np.float32(2.0) * dot, np.float32(0.0))
    want = np.argsort(D, axis=1, kind="stable")[:, :20]
    assert (gc == 20).all() and np.array_equal(gd, np.take_along_axis(D, want, 1))
    assert np.array_equal(gi.astype(np.int64), want)
    s.close()
