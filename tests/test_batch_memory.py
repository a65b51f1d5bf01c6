"""Device memory of a batch where memory is short: the label counts that phase 2 keeps wait for the first phase 2, so
that a batch that is only uploaded, seeded or proposed for fits where it fitted without them; and a phase 2 for whose
counts there is no room does without, to the same result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_kept_counts_where_memory_is_short():
    import torch

    from dmolp_b200 import graphs
    from dmolp_b200.batch import Batch, Instance

    n, k = 1_000_000, 40
    g = graphs.knn(n, 2, 8, seed=1)
    counts = 64 * n  # k >= 32: 32 labels of 16 bits per vertex
    lab0 = np.random.default_rng(1).integers(0, k, n).astype(np.int32)
    held = []

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def leave(size):
        """Device memory held until about `size` bytes are free."""
        for piece in (1 << 30, 1 << 26, 1 << 23):
            while free() > size + piece:
                held.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))

    def run(b):
        b.set_labels(lab0)
        res, _ = b.run("fixed", 4)
        return b.labels(), res[0]["edge_cut"]

    b = Batch(0)
    try:
        b.upload([Instance(graphs.knn(1000, 2, 8, seed=1), k)])  # the context, and one launch of each kind
        b.phase1(1000)
        b.run("fixed", 2)
        before = free()
        b.upload([Instance(g, k)])
        plenty = before - free()
        want, cut = run(b)
        assert before - free() < plenty + counts // 2  # they came with the upload
        b.upload([Instance(graphs.knn(1000, 2, 8, seed=1), k)])
        # less than 4 KB per vertex
        leave(3000 * n)
        before = free()
        b.upload([Instance(g, k)])
        short = before - free()
        assert short <= plenty - counts // 2
        b.phase1(1000)
        got, c = run(b)
        assert before - free() >= short + counts // 2
        assert np.array_equal(got, want) and c == cut
        # less than the counts
        b.upload([Instance(g, k)])
        leave(counts // 2)
        room = free()
        got, c = run(b)
        assert room - free() < counts // 4
        assert np.array_equal(got, want) and c == cut
    finally:
        held.clear()
        torch.cuda.empty_cache()
        b.close()
