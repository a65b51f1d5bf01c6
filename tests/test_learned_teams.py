"""The learned start on graphs that single blocks and lanes do not cover: hub rows searched by a whole team
(more than 4096 arcs), rows summed by a block of their own (more than 256), two components, graphs run by
clusters of CTAs.  Features, network and decoder against the oracle, at the tolerances of test_mpnn.py."""
import numpy as np
import pytest

from dmolp_b200 import graphs
from dmolp_b200.batch import Instance, union
from oracle import mpnn as M


def star_ring(n, hub, extra):
    """A ring over n vertices whose first vertex also joins `hub` others, and a path of `extra` vertices apart."""
    edges = [(i, (i + 1) % n) for i in range(n)] + [(0, i) for i in range(2, hub + 2)]
    return graphs.from_edges(n + extra, edges + [(n + i, n + i + 1) for i in range(extra - 1)])


def make(name):
    if name == "huge":
        return [Instance(star_ring(5200, 4500, 3), 5)]
    if name == "long":
        return [Instance(star_ring(300, 255, 2), 2), Instance(star_ring(700, 256, 0), 3), Instance(star_ring(900, 257, 5), 4)]
    return [Instance(graphs.knn(4500, 2, 6, seed=3), 11)]


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["huge", "long", "mesh"])
def test_learned_start_matches_oracle(name):
    from dmolp_b200.batch import Batch
    from dmolp_b200.learned import Proposal

    inst = make(name)
    b = Batch(0)
    b.upload(inst)
    m = Proposal(0)
    m.prepare_training(b)
    X = m.features(b)
    for i, it in enumerate(inst):
        ref = M.features(it.graph.offsets, it.graph.indices, it.k)
        np.testing.assert_allclose(X[b.vstart[i]:b.vstart[i + 1]], ref, rtol=2e-4, atol=2e-4)
    vstart, off, col, _ = union(inst)
    for i in range(len(inst)):
        col[off[vstart[i]]:off[vstart[i + 1]]] += vstart[i]
    rng = np.random.default_rng(5)
    P = (rng.standard_normal(M.num_params()) * 0.2).astype(np.float32)
    m.set_params(P)
    H = rng.standard_normal(X.shape).astype(np.float32)
    m.set_features(b, H)
    Z = m.forward(b)
    Zr, cache = M.forward(off, col, H, P)
    assert np.linalg.norm(Z - Zr) < 5e-3 * np.linalg.norm(Zr)
    R = rng.standard_normal(Z.shape).astype(np.float32)
    g, gr = m.backward(b, R), M.backward(off, col, cache, R, P)
    assert np.linalg.norm(g - gr) < 2e-2 * np.linalg.norm(gr)
    # the decoder on well-separated coordinates: every part's size within the splits' rounding
    Y = np.zeros(X.shape, np.float32)
    Y[:, :8] = rng.standard_normal((X.shape[0], 8)).astype(np.float32) * (8.0 ** -np.arange(8))
    st = m.decode(b, Y)
    assert not st.any()
    got = b.split(b.labels())
    for i, it in enumerate(inst):
        # set_features installed H: the coordinates are its random-walk columns plus Y
        a, z = b.vstart[i], b.vstart[i + 1]
        ref = M.decode(H[a:z], Y[a:z], it.k)
        assert np.mean(got[i] == ref) >= 0.97
        assert np.array_equal(np.bincount(got[i], minlength=it.k), np.bincount(ref, minlength=it.k))
    m.close()
    b.close()
