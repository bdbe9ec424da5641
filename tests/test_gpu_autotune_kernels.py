"""The autotuner times the warps per CTA only where the kernel has that choice."""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import synth

pytestmark = pytest.mark.gpu


def test_cta_searches_keep_the_default_warps():
    """Beams above 64 run a CTA per query, whose width follows from the batch:
    every value times the same there, so none may be chosen by chance."""
    X = synth.mixture(4000, 64, 16, seed=2)
    Q = synth.mixture(200, 64, 16, seed=2, stream=synth.STREAM_QUERY)
    adj = np.random.default_rng(2).integers(0, 4000, (4000, 32)).astype(np.uint32)
    ix = dg.DiskANN.from_graph(X, adj, 0)
    chosen = [ix.autotune(Q[:nq], 10, L, reps=2)["warps_per_cta"] for nq in (20, 200) for L in (65, 100, 200, 300)]
    assert chosen == [4] * len(chosen)
    assert ix.autotune(np.concatenate([Q] * 10), 10, 40, reps=2)["warps_per_cta"] in (1, 2, 4)
    ix.close()
