"""Graph construction over the range of alpha, against the CPU oracle: few and
many relaxed passes, and passes without end but for the largest float."""
import numpy as np
import pytest

import pydiskann_b200 as dg
from pydiskann_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [0.5, 1.3, 2.0, 7.9, 8.5, 100.0, float("inf")])
@pytest.mark.parametrize("shift,Lb", [(0.0, 40), (0.5, 40), (0.0, 200)])  # tensor-core, FMA, pools above 512
def test_vamana_alpha(oracle, alpha, shift, Lb):
    X = synth.mixture(900, 40, 8, seed=9) + np.float32(shift)
    adj, med = dg.build_graph(X, 24, Lb, alpha, seed=5)
    top = min(alpha, float(np.finfo(np.float32).max))  # the oracle's passes end too
    want, _ = oracle.build_vamana(X, 24, Lb, top, seed=5, medoid_id=med)
    assert np.array_equal(adj, want)
