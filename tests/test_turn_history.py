"""The turn between iterations in the launch-per-step form: every part's counts are in the history of every iteration,
the one that stops the run included.  (Its block's warps once could find the stop flag rewritten before they had
read it, and left without their share.)  Timed launches take this form on graphs of any size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [9, 300, 1024])
def test_counts_of_the_stopping_iteration(k):
    import oracle
    from dmolp_b200 import cabi, graphs
    from dmolp_b200.partitioner import Partitioner

    g = graphs.knn(6000, 3, 8, seed=k)
    lab0 = np.random.default_rng(k).integers(0, k, g.num_vertices).astype(np.int32)
    o = oracle.phase2(g.offsets, g.indices, lab0, k, "ref", 0)
    with Partitioner(0) as p:
        p.upload(g)
        assert p.lib.dmolp_set_profiling(p.ctx, 1) == cabi.DMOLP_OK
        for _ in range(12):
            p.set_labels(lab0)
            m = p.phase2(k, mode="ref")
            pen, cnt = p.history(k, m.iterations_run)
            assert m.iterations_run == o.res.iterations_run and m.stop_reason == o.res.stop_reason != 0
            assert np.array_equal(pen.view(np.int64), o.penalties.view(np.int64)) and np.array_equal(cnt, o.counts)
            assert np.array_equal(p.labels(), o.labels)
