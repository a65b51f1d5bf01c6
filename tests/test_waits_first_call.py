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
