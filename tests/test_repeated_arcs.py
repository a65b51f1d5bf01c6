"""Phase 1 on graphs that list an arc more than once: a seed whose row repeats neighbours of long rows, so that the
rows queued in pieces are each queued once however often they are listed.  Seeds and labels against the oracle."""
import numpy as np
import pytest

from dmolp_b200.graphs import Graph


def multigraph(n, first, repeats, long_row):
    """Vertex 0 joined `first` times to distinct vertices and `repeats` times to each of 1 and 2, whose rows have
    `long_row` more arcs each; a ring, and two hubs outside the first seed's ball.  Rows sorted, repeats kept."""
    rng = np.random.default_rng(repeats)
    half = n // 2
    parts = [np.stack([np.zeros(first, int), rng.choice(np.arange(3, half), first, replace=False)], 1)]
    for u in (1, 2):
        parts.append(np.tile([[0, u]], (repeats, 1)))
        parts.append(np.stack([np.full(long_row, u), rng.choice(np.arange(3, half), long_row, replace=False)], 1))
    for h in (half + 5, n - 7):
        nb = rng.choice(np.arange(half + 50, n - 50), first // 2, replace=False)
        parts.append(np.stack([np.full(nb.size, h), nb], 1))
    ring = np.arange(n)
    parts.append(np.stack([ring, (ring + 1) % n], 1))
    e = np.concatenate(parts)
    e = np.concatenate([e, e[:, ::-1]])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=n), out=off[1:])
    return Graph(off, e[:, 1].astype(np.int32))


def pieces_of_first_ball(g, once):
    """Row pieces of 512 arcs that the first seed's ball queues, and the queue's places."""
    deg = np.diff(g.offsets)
    row = g.indices[g.offsets[0]:g.offsets[1]]
    row = np.unique(row) if once else row
    d = deg[row[row != 0]]
    return int(((d[d > 512] + 511) // 512).sum()), g.num_arcs // 256 + 2


def test_each_row_once_fits_the_queue():
    g = multigraph(9000, 1500, 600, 700)
    n, cap = pieces_of_first_ball(g, True)
    assert n <= cap
    n, cap = pieces_of_first_ball(g, False)
    assert n > cap  # every occurrence would not


@pytest.mark.gpu
@pytest.mark.parametrize("k,theta", [(2, 10**6), (5, 40), (70, 7)])
def test_phase1_matches_oracle(k, theta):
    import oracle
    from dmolp_b200.partitioner import Partitioner

    g = multigraph(9000, 1500, 600, 700)
    o = oracle.phase1(g.offsets, g.indices, g.raw_deg(), k, theta)
    with Partitioner(0) as p:
        p.upload(g)
        for _ in range(2):  # the second call finds what the first left in the claim words
            m = p.phase1(k, theta)
            assert np.array_equal(m.seeds, o.seeds) and np.array_equal(p.labels(), o.labels)
            assert m.initial_edge_cut == o.res.initial_edge_cut
