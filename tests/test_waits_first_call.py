"""Bounded waits that run out in a call that is the first of its kind on a graph, when what the call would leave for
later ones is not there yet: the call returns DMOLP_ERR_CUDA, and the same context then gives the oracle's result
with the default limit.  No GPU fault is involved: a barrier that gives up only makes the blocks leave early."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gives_up(p, call):
    from dmolp_b200 import cabi
    from dmolp_b200.partitioner import DmolpError

    assert p.lib.dmolp_set_wait_limit(p.ctx, 1) == cabi.DMOLP_OK
    with pytest.raises(DmolpError) as e:
        call()
    assert e.value.code == cabi.DMOLP_ERR_CUDA and "gave up" in str(e.value)
    assert p.lib.dmolp_set_wait_limit(p.ctx, 0) == cabi.DMOLP_OK


@pytest.mark.parametrize("k", [16, 100])  # kept counts, every label's neighbours counted
def test_first_phase2(k):
    """The slot orders of the one-launch loop are built by a graph's first run; a larger graph before it leaves ids
    beyond this one's in the same buffers."""
    import oracle
    from dmolp_b200 import graphs
    from dmolp_b200.partitioner import Partitioner

    with Partitioner(0) as p:
        for g in (graphs.rmat(15, 8, seed=4), graphs.rmat(13, 8, seed=3)):
            lab0 = np.random.default_rng(k).integers(0, k, g.num_vertices).astype(np.int32)
            o = oracle.phase2(g.offsets, g.indices, lab0, k, "fixed", 6)
            p.upload(g)
            p.set_labels(lab0)
            for _ in range(2):
                gives_up(p, lambda: p.phase2(k, mode="fixed", iterations=6, records=False))
                p.set_labels(lab0)
            for _ in range(2):
                p.set_labels(lab0)
                m = p.phase2(k, mode="fixed", iterations=6, records=False)
                assert np.array_equal(p.labels(), o.labels)
                assert m.edge_cut == o.res.edge_cut and m.traversed_edges == o.res.te_total


@pytest.mark.parametrize("kind,k", [("seeds", 9), ("growth", 1), ("hubs", 9)])
def test_first_phase1(kind, k):
    """The seed search; the growth alone (one part needs no search), with the metrics of what it left; the degree
    statistics of a graph whose hub list starts on the device."""
    import oracle
    from dmolp_b200 import graphs
    from dmolp_b200.partitioner import Partitioner

    g = graphs.rmat(17 if kind == "hubs" else 13, 8, seed=5)
    o = oracle.phase1(g.offsets, g.indices, g.raw_deg(), k, 50)
    with Partitioner(0) as p:
        p.upload(g)
        for _ in range(2):
            gives_up(p, lambda: p.phase1(k, 50))
            m = p.phase1(k, 50)
            assert np.array_equal(m.seeds, o.seeds) and np.array_equal(p.labels(), o.labels)
            assert m.rounds == o.res.rounds and m.traversed_edges == o.res.te


def test_seed_and_growth_entries():
    import ctypes

    import oracle
    from dmolp_b200 import graphs
    from dmolp_b200.partitioner import Partitioner

    g, k = graphs.barabasi_albert(5000, 5, seed=2), 12
    o = oracle.phase1(g.offsets, g.indices, g.raw_deg(), k, 30)
    hubs = np.argsort(-g.raw_deg(), kind="stable")[:800].astype(np.int32)
    first = int(hubs[0])
    with Partitioner(0) as p:
        p.upload(g)

        def find():
            out, n = np.empty(k, np.int32), ctypes.c_int32()
            p._check(p.lib.dmolp_find_seeds(p.ctx, k, first, hubs.ctypes.data, hubs.size, out.ctypes.data, ctypes.byref(n)))
            return out[:n.value].tolist()

        def grow(seeds):
            s, r = np.array(seeds, np.int32), ctypes.c_int32()
            p._check(p.lib.dmolp_expand_partitions(p.ctx, k, 30, s.ctypes.data, s.size, ctypes.byref(r)))
            return r.value

        want = find()
        gives_up(p, find)
        assert find() == want
        assert grow(o.seeds) == o.res.rounds
        gives_up(p, lambda: grow(o.seeds))
        assert grow(o.seeds) == o.res.rounds and np.array_equal(p.labels(), o.labels)


def test_first_features_of_a_large_graph():
    """The anchor searches of a graph worth more CTAs than a cluster meet at barriers of their own."""
    from dmolp_b200 import cabi, graphs
    from dmolp_b200.batch import Batch, Instance
    from dmolp_b200.learned import Proposal
    from dmolp_b200.partitioner import DmolpError

    b = Batch(0)
    b.upload([Instance(graphs.barabasi_albert(80_000, 5, seed=3), 7), Instance(graphs.knn(900, 2, 6, seed=1), 3)])
    ref, m = Proposal(0), Proposal(0)
    try:
        want = ref.features(b)
        for _ in range(2):
            assert m.lib.dmolp_mpnn_set_wait_limit(m.h, 1) == cabi.DMOLP_OK
            with pytest.raises(DmolpError) as e:
                m.features(b)
            assert e.value.code == cabi.DMOLP_ERR_CUDA and "timed out" in str(e.value)
            assert m.lib.dmolp_mpnn_set_wait_limit(m.h, 0) == cabi.DMOLP_OK
            np.testing.assert_allclose(m.features(b), want, rtol=1e-5, atol=1e-5)  # (sums over chunks in any order)
    finally:
        ref.close()
        m.close()
        b.close()
