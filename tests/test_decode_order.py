"""The decoder's labels of a graph depend on the graph and its coordinates, not on the batch it is in: a team of CTAs
sums a part's mean and covariance in an order that the graph and the part alone decide.  The coordinates are closed under
exchange and signs of two axes, so the principal axis is decided by the last bits of the sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def coordinates(n, seed):
    rng = np.random.default_rng(seed)
    q = rng.standard_normal((n // 8, 2)).astype(np.float32)
    q = np.concatenate([q, q[:, ::-1]])
    q = np.concatenate([q * np.float32(s) for s in ([1, 1], [1, -1], [-1, 1], [-1, -1])])
    Y = np.zeros((n, 16), np.float32)
    Y[:q.shape[0], :2] = q[rng.permutation(q.shape[0])]
    return Y


@pytest.mark.parametrize("n,k", [(255, 3), (4097, 2), (20011, 9), (70001, 64)])
def test_same_labels_in_any_batch(n, k):
    from dmolp_b200 import graphs
    from dmolp_b200.batch import Batch, Instance
    from dmolp_b200.learned import Proposal

    g, Y = graphs.knn(n, 2, 6, seed=n), coordinates(n, n)
    others = [graphs.knn(m, 2, 6, seed=m) for m in (300_000, 40_000, 6000, 700)]
    got = []
    for before, after in (([], []), (others[:1], []), (others[1:3], others[3:]), ([], others), (others[3:] * 40, [])):
        inst = [Instance(x, 5) for x in before] + [Instance(g, k)] + [Instance(x, 7) for x in after]
        b, m = Batch(0), Proposal(0)
        try:
            b.upload(inst)
            m.set_features(b, np.zeros((b.num_vertices, 16), np.float32))
            E = np.random.default_rng(3).standard_normal((b.num_vertices, 16)).astype(np.float32)
            i = len(before)
            E[b.vstart[i]:b.vstart[i + 1]] = Y
            assert m.decode(b, E)[i] == 0
            got.append(b.split(b.labels())[i])
        finally:
            m.close()
            b.close()
    size = np.bincount(got[0], minlength=k)
    assert size.min() > 0 and size.sum() == n
    for x in got[1:]:
        assert np.array_equal(x, got[0])
