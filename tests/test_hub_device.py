"""The hub list whose first partitions run on the device: its order, ties included, against the oracle's std::sort,
through the seeds it decides (the completion takes unused hubs in order), on graphs just above the device path's size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ties(n, centres, leaves):
    """A ring, and every centre joined to the same number of vertices: hubs of equal degree."""
    from dmolp_b200.graphs import Graph

    rng = np.random.default_rng(centres)
    c = rng.choice(n, centres, replace=False)
    u = np.repeat(c, leaves)
    v = (u + 2 + np.tile(np.arange(leaves), centres) * 7) % n
    ring = np.arange(n)
    e = np.concatenate([np.stack([u, v], 1), np.stack([ring, (ring + 1) % n], 1)])
    e = np.unique(np.concatenate([e, e[:, ::-1]]), axis=0)
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=n), out=off[1:])
    return Graph(off, e[:, 1].astype(np.int32))


@pytest.mark.parametrize("kind", ["rmat17", "rmat18", "ties", "few"])
def test_seeds_match_oracle(kind):
    import oracle
    from dmolp_b200 import graphs
    from dmolp_b200.partitioner import Partitioner

    g = {"rmat17": lambda: graphs.rmat(17, 8, seed=5), "rmat18": lambda: graphs.rmat(18, 4, seed=6),
         "ties": lambda: _ties(200_003, 2000, 60), "few": lambda: _ties(131_072, 40, 3000)}[kind]()
    k = 700
    with Partitioner(0) as p:
        p.upload(g)
        m = p.phase1(k, 10**6)
        labels = p.labels()
    o = oracle.phase1(g.offsets, g.indices, g.raw_deg(), k, 10**6)
    assert np.array_equal(m.seeds, o.seeds)
    assert np.array_equal(labels, o.labels)
