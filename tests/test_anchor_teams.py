"""Anchor searches by teams of a cooperative launch, graphs worth more CTAs than a cluster: alone, two side by side,
and next to a small graph on a cluster.  Features against the oracle at the tolerances of test_mpnn.py."""
import numpy as np
import pytest

from dmolp_b200 import graphs
from dmolp_b200.batch import Instance
from oracle import mpnn as M


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(80_000,), (50_000, 45_000), (90_000, 1200)])
def test_features_match_oracle(sizes):
    from dmolp_b200.batch import Batch
    from dmolp_b200.learned import Proposal

    inst = [Instance(graphs.barabasi_albert(n, 5, seed=n), 7) for n in sizes]
    b = Batch(0)
    b.upload(inst)
    m = Proposal(0)
    X = m.features(b)
    for i, it in enumerate(inst):
        ref = M.features(it.graph.offsets, it.graph.indices, it.k)
        np.testing.assert_allclose(X[b.vstart[i]:b.vstart[i + 1]], ref, rtol=2e-4, atol=2e-4)
    m.close()
    b.close()
