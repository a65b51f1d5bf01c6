"""Phase 2 with a launch per step on graphs that would take the one-launch loop: the form that every larger graph runs,
held to the oracle by the tests of small graphs (imported here and run again with the option on), by the stopping
rules, and by its first run on a graph (launched), second (captured) and third (replayed)."""
import numpy as np
import pytest

import oracle
from test_gpu_parity import test_phase2_matches_reference, test_random_cases_against_oracle  # noqa: F401
from test_hub_counts import (hub_graph, part, test_graph_without_hubs_after_one_with_hubs,  # noqa: F401
                             test_hub_decisions_match_oracle, test_hub_decisions_reference_stopping_rules)
from test_lp_loop import test_loop_matches_oracle  # noqa: F401
from test_symmetry import edit_rows
from test_waits import test_selection_barrier_gives_up_and_context_recovers  # noqa: F401
from test_waits_first_call import test_first_phase2  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def steps():
    """Every context of this module takes a launch per step."""
    from dmolp_b200.partitioner import Partitioner

    init = Partitioner.__init__

    def with_steps(self, *args, **kw):
        init(self, *args, **kw)
        self.set_lp_steps(True)

    with pytest.MonkeyPatch.context() as mp:
        mp.setattr(Partitioner, "__init__", with_steps)
        yield


def check(p, g, lab0, k, mode, iters, cap, o):
    p.set_labels(lab0)
    m = p.phase2(k, mode=mode, iterations=iters, cap=cap)
    assert np.array_equal(p.labels(), o.labels)
    assert m.iterations_run == o.res.iterations_run and m.stop_reason == o.res.stop_reason
    assert m.edge_cut == o.res.edge_cut and m.traversed_edges == o.res.te_total
    for r, s in zip(m.records, o.records):
        assert (r.window, r.changes, r.edge_cut) == (s.window, s.changes, s.edge_cut), r.iteration
    pen, cnt = p.history(k, m.iterations_run)
    assert np.array_equal(pen.view(np.int64), o.penalties.view(np.int64)) and np.array_equal(cnt, o.counts)


@pytest.mark.parametrize("k,cap", [(8, "ref"), (40, "full"), (65, "ref"), (100, "full"), (1000, "ref")])
@pytest.mark.parametrize("mode", ["ref", "fixed"])
def test_first_captured_and_replayed_run(k, cap, mode):
    from dmolp_b200.partitioner import Partitioner

    g = hub_graph(seed=k)
    lab0 = np.random.default_rng(k).integers(0, k, g.num_vertices).astype(np.int32)
    o = oracle.phase2(g.offsets, g.indices, lab0, k, mode, 9, cap)
    with Partitioner(0) as p:
        p.upload(g)
        assert p.symmetric()
        for _ in range(3):
            before = p.kernel_launches()
            check(p, g, lab0, k, mode, 9, cap, o)
            assert p.kernel_launches() - before > 4 * o.res.iterations_run


def stopping_case(reason, k):
    from dmolp_b200 import graphs

    if reason == 1:  # nothing on a boundary
        g = graphs.knn(3000, 2, 6, seed=1)
        return g, np.zeros(g.num_vertices, np.int32), k
    if reason == 2:  # two cliques joined by an edge, a label each: a boundary, and no vertex to gain by moving
        n = 40
        e = [(i, j) for c in (0, n) for i in range(c, c + n) for j in range(i + 1, c + n)] + [(0, n)]
        return graphs.from_edges(2 * n, e), np.repeat([0, 1], n).astype(np.int32), k
    g = graphs.barabasi_albert(9000, 6, seed=1)  # self-loops on every seventh vertex
    g = edit_rows(g, {v: sorted(set(g.indices[g.offsets[v]:g.offsets[v + 1]].tolist()) | {v}) for v in range(0, 9000, 7)})
    return g, np.random.default_rng(3).integers(0, k, 9000).astype(np.int32), k


@pytest.mark.parametrize("reason,k", [(1, 4), (2, 2), (2, 70), (3, 16)])
def test_stopping_rules(reason, k):
    from dmolp_b200.partitioner import Partitioner

    g, lab0, k = stopping_case(reason, k)
    o = oracle.phase2(g.offsets, g.indices, lab0, k, "ref", 0)
    assert o.res.stop_reason == reason
    with Partitioner(0) as p:
        p.upload(g)
        for on in (True, True, True, False, True):  # and after a run of the other form
            p.set_lp_steps(on)
            check(p, g, lab0, k, "ref", 0, "ref", o)
