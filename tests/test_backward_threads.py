"""Networks of several host threads: some batches have rows that the backward aggregation stages in shared memory, the
others have none.  Each call's launch has to be right whatever the other threads launch in between."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_backward_in_threads():
    from dmolp_b200 import graphs
    from dmolp_b200.batch import Batch, Instance
    from dmolp_b200.learned import Proposal

    star = graphs.from_edges(400, [(0, i) for i in range(1, 400)])  # a row of more than 256 arcs
    failures = []

    def work(g):
        b, m = Batch(0), Proposal(0)
        try:
            b.upload([Instance(g, 4)])
            m.prepare_training(b)
            rng = np.random.default_rng(g.num_vertices)
            m.set_params((rng.standard_normal(m.n) * 0.2).astype(np.float32))
            m.set_features(b, rng.standard_normal((b.num_vertices, 16)).astype(np.float32))
            m.forward(b)
            R = rng.standard_normal((b.num_vertices, 16)).astype(np.float32)
            start.wait(60)
            for _ in range(1000):
                m.backward(b, R)
        except Exception as e:  # noqa: BLE001  (reported by the test)
            failures.append(repr(e))
        finally:
            m.close()
            b.close()

    jobs = [star, star] + [graphs.knn(200 + i, 2, 6, seed=i) for i in range(6)]
    start = threading.Barrier(len(jobs))
    threads = [threading.Thread(target=work, args=(g,)) for g in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
