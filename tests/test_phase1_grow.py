"""Phase 1's two launches (seeds, growth) against the oracle where their branches meet: rows at the split into
pieces, frontiers at theta, empty frontiers, parts without a seed, more labels than the shared histograms hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, edges):
    from dmolp_b200.graphs import Graph

    e = np.unique(np.concatenate([edges, edges[:, ::-1]]), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=n), out=off[1:])
    return Graph(off, e[:, 1].astype(np.int32))


def _stars(n, centres, leaves, seed):
    """Centre i is joined to leaves[i] vertices, plus a sparse random graph on all of them."""
    rng = np.random.default_rng(seed)
    parts = [np.stack([np.full(m, c), rng.choice(n, m, replace=False)], 1) for c, m in zip(centres, leaves)]
    parts.append(rng.integers(0, n // 2, (n, 2)))  # the upper half is reached through the stars only
    return _graph(n, np.concatenate(parts))


@pytest.mark.parametrize("k,theta", [(1, 1), (2, 7), (5, 100), (64, 3), (65, 40), (100, 10**6)])
@pytest.mark.parametrize("n,leaves", [(40, (3,)), (1500, (31, 32, 33, 511, 512, 513)), (6000, (1024, 1025, 5000))])
def test_growth_matches_oracle(n, leaves, k, theta):
    import oracle
    from dmolp_b200.partitioner import Partitioner

    if k > n:
        pytest.skip("more parts than vertices")
    g = _stars(n, range(len(leaves)), leaves, seed=n + k)
    with Partitioner(0) as p:
        p.upload(g)
        m = p.phase1(k, theta)
        labels = p.labels()
    o = oracle.phase1(g.offsets, g.indices, g.raw_deg(), k, theta)
    assert np.array_equal(labels, o.labels)
    assert m.initial_edge_cut == o.res.initial_edge_cut
