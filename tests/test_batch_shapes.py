"""A batch's launch shape is the one asked for, whatever shape ran before it: the teams that a shape's residency gives
the graphs are part of what is captured for it."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grids(b, shape, path):
    """(kernel, blocks) of the phase-2 launches of one run, sorted."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.init()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        b.run("fixed", 4, tuning=shape)
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    ev = json.load(open(path))["traceEvents"]
    out = [(e["name"].split("<")[0], tuple(e["args"]["grid"])) for e in ev
           if e.get("cat") == "kernel" and "k_batch_lp" in e["name"]]
    if not out:
        pytest.skip("no kernel records from the profiler here")
    return sorted(out)


def test_shape_after_another_shape(tmp_path):
    from dmolp_b200 import graphs
    from dmolp_b200.batch import Batch, Instance

    inst = [Instance(graphs.knn(n, 2, 6, seed=n), 6) for n in (60_000, 20_000, 9000, 5000, 3000, 2000, 1000, 500)]
    shapes = [{"block_threads": 256, "thread_row_max": 8, "blocks_per_sm": s} for s in (1, 4)]
    fresh = []
    for s in shapes:
        b = Batch(0)
        b.upload(inst)
        fresh.append(grids(b, s, tmp_path / "t.json"))
        b.close()
    assert fresh[0] != fresh[1]  # four times the slots: larger teams
    b = Batch(0)
    b.upload(inst)
    lab0 = [np.random.default_rng(i).integers(0, 6, it.graph.num_vertices).astype(np.int32) for i, it in enumerate(inst)]
    labels = []
    for s, want in list(zip(shapes, fresh)) + list(zip(shapes, fresh)):
        b.set_labels(lab0)
        assert grids(b, s, tmp_path / "t.json") == want
        labels.append(b.labels())
    assert all(np.array_equal(x, labels[0]) for x in labels)
    b.close()
