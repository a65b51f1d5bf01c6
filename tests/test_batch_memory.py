"""Device memory of a batch: the label counts that phase 2 keeps are allocated by the first phase 2, so that a batch
that is only uploaded, seeded or proposed for fits where it fitted without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_kept_counts_come_with_phase2():
    import torch

    from dmolp_b200 import graphs
    from dmolp_b200.batch import Batch, Instance

    n = 1_000_000
    g = graphs.knn(n, 2, 8, seed=1)
    counts = 64 * n  # k >= 32: 32 labels of 16 bits per vertex

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    b = Batch(0)
    b.upload([Instance(graphs.knn(1000, 2, 8, seed=1), 40)])  # the context, and one launch of each kind
    b.phase1(1000)
    b.run("fixed", 2)
    before = free()
    b.upload([Instance(g, 40)])
    b.phase1(1000)
    used = before - free()
    # offsets, ids, and fewer than 24 words of 4 bytes per vertex; allocations rounded up to 2 MB each
    assert used < 8 * n + 4 * g.num_arcs + 24 * 4 * n < used + counts
    b.run("fixed", 2)
    assert before - free() >= used + counts
    b.upload([Instance(graphs.knn(1000, 2, 8, seed=1), 40)])
    assert free() > before - (32 << 20)  # given back with the batch
    b.close()
