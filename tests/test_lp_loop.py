"""The LP loop in one launch against the oracle, iteration by iteration, where its steps change form: rows at one
lane's and one piece's length and above the hub bound, labels beyond the 32 scored ones, every label scored, one
record per block and several per warp, runs that stop by themselves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stars(n, leaves, seed):
    """Vertex i is joined to leaves[i] others, on top of a sparse random graph; symmetric, no loops."""
    from dmolp_b200.graphs import Graph

    rng = np.random.default_rng(seed)
    parts = [np.stack([np.full(m, c), rng.choice(n, m, replace=False)], 1) for c, m in enumerate(leaves)]
    parts.append(rng.integers(0, n, (3 * n, 2)))
    e = np.concatenate(parts)
    e = np.unique(np.concatenate([e, e[:, ::-1]]), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(e[:, 0], minlength=n), out=off[1:])
    return Graph(off, e[:, 1].astype(np.int32))


@pytest.mark.parametrize("n,leaves", [(60, (31, 33)), (3000, (15, 17, 32, 255, 256, 257, 512, 513)),
                                      (90000, (4096, 4097, 9000))])
@pytest.mark.parametrize("k,cap,mode", [(2, "ref", "fixed"), (7, "ref", "ref"), (32, "full", "fixed"), (33, "ref", "fixed"),
                                        (33, "full", "ref"), (200, "full", "fixed"), (1024, "ref", "fixed")])
def test_loop_matches_oracle(n, leaves, k, cap, mode):
    import oracle
    from dmolp_b200.partitioner import Partitioner

    g = _stars(n, leaves, seed=n)
    lab0 = np.random.default_rng(k).integers(0, k, n).astype(np.int32)
    with Partitioner(0) as p:
        p.upload(g)
        assert p.symmetric()
        for _ in range(2):  # the second run reuses the slot orders
            p.set_labels(lab0)
            m = p.phase2(k, mode=mode, iterations=7, cap=cap)
            labels = p.labels()
        pen, cnt = p.history(k, m.iterations_run)
    o = oracle.phase2(g.offsets, g.indices, lab0, k, mode, 7, cap)
    assert m.iterations_run == o.res.iterations_run and m.stop_reason == o.res.stop_reason
    for r, s in zip(m.records, o.records):
        assert (r.window, r.changes, r.edge_cut) == (s.window, s.changes, s.edge_cut), r.iteration
    assert np.array_equal(labels, o.labels)
    assert np.array_equal(pen.view(np.int64), o.penalties.view(np.int64)) and np.array_equal(cnt, o.counts)
    assert m.traversed_edges == o.res.te_total
