"""The partitioner's workloads: what is run, on what sizes, and what each cannot do without.

Kinds of work, each through the public entry points (`Partitioner`, `Batch`, `Proposal`):

  metrics    cut and part sizes of a labelling on the resident graph (the reference's -m metrics pass)
  lp         phase 2 alone on a resident graph, from phase-1 labels kept on the device
  partition  the whole call on a graph in host arrays: upload, phase 1, phase 2, labels back
  text       adjacency text in device memory parsed into the resident graph, then phase 1
  batch      many small graphs at once: batched phase 1, batched phase 2, labels back
  learned    the same with the learned start: proposal, phase 1 where its gate declines, phase 2
  propose    the learned start on one graph with the gate ignored: features, network, decoder
  train      one training step of the proposal's gate: forward, backward, weight update
"""
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from dmolp_b200 import graphs
from dmolp_b200.batch import Batch, Instance, union
from dmolp_b200.graphs import Graph
from dmolp_b200.learned import WEIGHTS, Proposal
from dmolp_b200.partitioner import Partitioner


def listed():
    return [
        # scoring a partition that another tool made: the smallest call, a reduction over one small mesh
        dict(name="metrics-knn3d-55k", kind="metrics", graph="knn3d", n=55476, deg=12, k=8, theta=1000),
        # refining a small mesh partition: launches and latency decide
        dict(name="lp-knn3d-55k-k8", kind="lp", graph="knn3d", n=55476, deg=12, k=8, theta=1000, mode="fixed",
             iterations=20, cap="ref"),
        # every label scored (more than 32), run to convergence on a preferential-attachment network
        dict(name="lp-ba-150k-k100-full", kind="lp", graph="ba", n=150001, deg=6, k=100, theta=1000, mode="ref",
             iterations=0, cap="full"),
        # the large social-network graph of the benchmark: scale 22, 128 M arcs, k = 32, 30 iterations
        dict(name="lp-rmat-4m-k32", kind="lp", graph="rmat", n=1 << 22, deg=16, k=32, theta=10000, mode="fixed",
             iterations=30, cap="ref"),
        # the whole call on a small planar mesh: set-up, rounds and host steps weigh most
        dict(name="partition-knn2d-5k-k8", kind="partition", graph="knn2d", n=5003, deg=10, k=8, theta=100),
        # the whole call on a skewed graph of a million vertices (an odd count), to convergence
        dict(name="partition-rmat-1m-k16", kind="partition", graph="rmat", n=1_000_003, deg=16, k=16, theta=10000),
        # a graph arriving as text (100 MB) through the caller's own I/O path, then its first partition
        dict(name="text-rmat-512k-k32", kind="text", graph="rmat", n=1 << 19, deg=16, k=32, theta=10000),
        # a minibatch of the mixed workload: few graphs of very different sizes
        dict(name="batch-64-mixed", kind="batch", count=64, vmin=1000, vmax=200_000, theta=1000),
        # many small graphs of like size
        dict(name="batch-512-small", kind="batch", count=512, vmin=1000, vmax=10_000, theta=1000),
        # the mixed workload with the learned start
        dict(name="learned-64-mixed", kind="learned", count=64, vmin=1000, vmax=200_000, theta=1000),
        # the learned start on one large graph (where its gate pays: skewed graphs)
        dict(name="propose-rmat-1m-k32", kind="propose", graph="rmat", n=1 << 20, deg=16, k=32),
        # a training minibatch of the proposal network
        dict(name="train-64-mixed", kind="train", count=64, vmin=1000, vmax=50_000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, largest):
    fam = rng.choice(("rmat", "rmat", "ba", "knn2d", "knn3d"))
    if fam == "rmat":
        return dict(graph=fam, n=_log_uniform(rng, 2000, largest), deg=rng.randint(8, 16))
    if fam == "ba":
        return dict(graph=fam, n=_log_uniform(rng, 2000, min(largest, 400_000)), deg=rng.randint(4, 8))
    return dict(graph=fam, n=_log_uniform(rng, 2000, min(largest, 300_000)), deg=rng.randint(8, 14))


def draw(rng):
    kind = rng.choice(("metrics", "lp", "lp", "lp", "partition", "partition", "text", "batch", "batch", "learned",
                       "propose", "train"))
    if kind in ("batch", "learned", "train"):
        vmin = 1000
        vmax = _log_uniform(rng, 2000, 50_000 if kind == "train" else 200_000)
        mean = (vmax - vmin) / math.log(vmax / vmin)
        count = _log_uniform(rng, 4, max(8, min(512, int(2_200_000 / mean))))
        c = dict(kind=kind, count=count, vmin=vmin, vmax=vmax)
        return c if kind == "train" else dict(c, theta=rng.choice((100, 1000, 3000)))
    c = dict(kind=kind, **_draw_graph(rng, {"metrics": 4_000_000, "lp": 4_000_000, "partition": 1_000_000,
                                            "text": 500_000, "propose": 1_000_000}[kind]))
    c["k"] = rng.choice((2, 4, 8, 12, 16, 24, 32, 48, 64)) if rng.random() < 0.8 else rng.randint(2, 128)
    if kind == "propose":
        c["k"] = min(c["k"], 64)
        return c
    c["theta"] = rng.choice((100, 1000, 10000)) if c["n"] <= 50_000 else rng.choice((1000, 10000))
    if kind == "lp":
        c["mode"] = rng.choice(("ref", "fixed"))
        c["iterations"] = rng.randint(5, 40) if c["mode"] == "fixed" else 0
        c["cap"] = rng.choice(("ref", "ref", "full"))
    return c


# ------------------------------------------------------------------------------------------------ inputs
def _rmat(n, edge_factor, seed):
    """Symmetrised R-MAT (0.57, 0.19, 0.19, 0.05) without loops and duplicates, ids permuted, made on the
    device; n vertices of the next power of two are kept.  (offsets, indices) device tensors."""
    scale = max(1, (n - 1).bit_length())
    m = edge_factor << scale
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.zeros(m, dtype=torch.int32, device="cuda")
    v = torch.zeros(m, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, device="cuda", generator=gen)
        hi = r >= 0.76
        u.mul_(2).add_(hi)
        v.mul_(2).add_(((r >= 0.57) & ~hi) | (r >= 0.95))
    perm = torch.randperm(1 << scale, device="cuda", generator=gen)
    u, v = perm[u], perm[v]
    keep = (u != v) & (u < n) & (v < n)
    u, v = u[keep], v[keep]
    keys = torch.unique(torch.cat([u * n + v, v * n + u]))
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(torch.div(keys, n, rounding_mode="floor"), minlength=n), 0, out=off[1:])
    return off, (keys % n).int()


def _graph(case, seed):
    n, fam = case["n"], case["graph"]
    if fam == "rmat":
        off, col = _rmat(n, case["deg"], seed)
        return Graph(off.cpu().numpy(), col.cpu().numpy())
    if fam == "ba":
        return graphs.barabasi_albert(n, case["deg"], seed=seed + 1)
    return graphs.knn(n, int(fam[3]), case["deg"], seed=seed + 1)


def _text(off, col, n):
    """The reference's adjacency text of a CSR on the device: a header line with the vertex count, then one
    line of space-separated neighbour ids per vertex.  uint8 device tensor."""
    head = torch.tensor(list(b"%d\n" % n), dtype=torch.uint8, device="cuda")
    digits = torch.ones_like(col, dtype=torch.int64)
    for d in range(1, 10):
        digits += col >= 10**d
    ends = torch.zeros(col.numel() + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(digits + 1, 0, out=ends[1:])
    deg = off[1:] - off[:-1]
    row_bytes = ends[off[1:]] - ends[off[:-1]] + (deg == 0)
    row_end = head.numel() + torch.cumsum(row_bytes, 0)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    start = (row_end - row_bytes)[row] + ends[:-1] - ends[off[:-1]][row]
    out = torch.full((int(row_end[-1]),), 32, dtype=torch.uint8, device="cuda")
    out[: head.numel()] = head
    out[row_end - 1] = 10
    for d in range(10):
        has = digits > d
        if not bool(has.any()):
            break
        out[(start + digits - 1 - d)[has]] = (48 + torch.div(col[has], 10**d, rounding_mode="floor") % 10).to(torch.uint8)
    return out


class _DeviceArray:
    """A device buffer of the library as an array for torch, which keeps its owner alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 2}


def _device_labels(p):
    import ctypes

    ptr = ctypes.c_void_p()
    p._check(p.lib.dmolp_device_labels(p.ctx, ctypes.byref(ptr)))
    return torch.as_tensor(_DeviceArray(p, ptr.value, p.num_vertices), device="cuda")


def _instances(case, seed):
    """The batched workload's mix: vertex counts log-uniform in [vmin, vmax], half geometric k-NN graphs (2-D
    or 3-D points, 8 to 14 neighbours), half preferential attachment (4 to 8), 2 to 64 parts.  Sizes and part
    counts are the case's, the graphs the seed's."""
    rng = np.random.default_rng([case["count"], case["vmin"], case["vmax"]])
    sizes = np.exp(rng.uniform(math.log(case["vmin"]), math.log(case["vmax"]), case["count"])).round().astype(int)
    parts, dims = rng.integers(2, 65, case["count"]), rng.integers(2, 4, case["count"])
    knn, m = rng.integers(8, 15, case["count"]), rng.integers(4, 9, case["count"])
    seeds = np.random.default_rng(seed).integers(1, 2**31 - 1, case["count"])

    def make(i):
        n, s = int(sizes[i]), int(seeds[i])
        g = graphs.barabasi_albert(n, int(m[i]), seed=s) if i % 2 else graphs.knn(n, int(dims[i]), int(knn[i]), seed=s)
        return Instance(g, int(parts[i]))

    with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        return list(ex.map(make, range(case["count"])))


def _train_inputs(case, seed):
    """The union CSR of a batch, input features of the network's layout (degree / mean degree, log degree,
    eight standardised coordinates, k / 64), gate targets (one in six positive)."""
    arrays = union(_instances(case, seed))
    rng = np.random.default_rng(seed)
    vstart, off, _, parts = arrays
    deg = np.diff(off).astype(np.float32)
    X = np.zeros((int(vstart[-1]), 16), np.float32)
    X[:, 1] = np.log1p(deg)
    X[:, 2:10] = rng.standard_normal((X.shape[0], 8), np.float32)
    for i, k in enumerate(parts):
        a, z = vstart[i], vstart[i + 1]
        X[a:z, 0] = deg[a:z] / max(1e-6, float(deg[a:z].mean()))
        X[a:z, 10] = k / 64.0
    y = (rng.random(len(parts)) < 1 / 6).astype(np.float32)
    return arrays, X, y


_LR = 1e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "learned"):
        inst = _instances(case, seed)
        b = Batch(0)
        b.upload(inst)
        return dict(case=case, b=b, model=Proposal(0, WEIGHTS) if kind == "learned" else None)
    if kind == "train":
        arrays, X, y = _train_inputs(case, seed)
        b = Batch(0)
        b.upload(arrays=arrays)
        model = Proposal(0, WEIGHTS)
        model.prepare_training(b)
        model.features(b, copy=False)
        pinned = torch.from_numpy(X).pin_memory()
        return dict(case=case, b=b, model=model, X=pinned.numpy(), y=y)
    if kind == "propose":
        b = Batch(0)
        b.upload([Instance(_graph(case, seed), case["k"])])
        return dict(case=case, b=b, model=Proposal(0, WEIGHTS))
    p = Partitioner(0)
    if kind == "text":
        if case["graph"] == "rmat":
            off, col = _rmat(case["n"], case["deg"], seed)
        else:
            g = _graph(case, seed)
            off, col = torch.from_numpy(g.offsets).cuda(), torch.from_numpy(g.indices).cuda()
        return dict(case=case, p=p, text=_text(off, col, case["n"]))
    g = _graph(case, seed)
    if kind == "partition":
        return dict(case=case, p=p, g=g)
    p.upload(g)
    p.phase1(case["k"], case["theta"])
    if kind == "lp":
        p._check(p.lib.dmolp_labels_save(p.ctx))
    return dict(case=case, p=p, labels=_device_labels(p))


# ------------------------------------------------------------------------------------------------ passes
def _phase1_outputs(m):
    return dict(cut=m.initial_edge_cut, vertices=np.array(m.partition_vertex_counts),
                edges=np.array(m.partition_edge_counts), seeds=np.array(m.seeds), rounds=m.rounds)


def _phase2_outputs(m):
    return dict(cut=m.edge_cut, vertex_balance=m.vertex_balance, edge_balance=m.edge_balance,
                iterations=m.iterations_run, traversed=m.traversed_edges)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "metrics":
        cut, vc, ec = state["p"].metrics(case["k"])
        return dict(cut=cut, vertices=vc, edges=ec)
    if kind == "lp":
        p = state["p"]
        p._check(p.lib.dmolp_labels_restore(p.ctx))
        m = p.phase2(case["k"], mode=case["mode"], iterations=case["iterations"], cap=case["cap"], records=False)
        return dict(_phase2_outputs(m), labels=state["labels"])
    if kind == "partition":
        p = state["p"]
        p.upload(state["g"])
        m1 = p.phase1(case["k"], case["theta"])
        m2 = p.phase2(case["k"], records=False)
        return dict(phase1=_phase1_outputs(m1), phase2=_phase2_outputs(m2), labels=p.labels())
    if kind == "text":
        p = state["p"]
        info = p.upload_adjtext(state["text"])
        m1 = p.phase1(case["k"], case["theta"])
        return dict(arcs=info["num_arcs"], phase1=_phase1_outputs(m1), labels=p.labels())
    b, model = state["b"], state["model"] if "model" in state else None
    if kind == "train":
        model.set_features(b, state["X"])
        loss = model.train_gate(b, state["y"], _LR)
        return dict(params=model.params(), loss=np.float32(loss))
    if kind == "propose":
        model.features(b, copy=False)
        model.forward(b, copy=False)
        status = model.decode(b)
        return dict(status=status, labels=b.labels())
    status = np.ones(case["count"], np.int32)
    if kind == "learned":
        status = model.propose(b)
    if kind == "batch":
        b.phase1(case["theta"])
    elif status.any():
        b.phase1(case["theta"], only=status != 0)
    res, _ = b.run("ref")
    return dict(status=status, labels=b.labels(), cut=np.array([r["edge_cut"] for r in res]),
                iterations=np.array([r["iterations_run"] for r in res]),
                balance=np.array([r["vertex_balance"] for r in res]))


# ------------------------------------------------------------------------------------------------ bounds
_WIDTHS = ((32, 64), (128, 64), (128, 16))  # the network's layers: inputs (own and neighbours'), outputs


def _sizes(case):
    """Vertices and arcs, from the generators' parameters."""
    if "count" in case:
        nv = case["count"] * (case["vmax"] - case["vmin"]) / math.log(case["vmax"] / case["vmin"])
        return nv, 12.4 * nv
    n = case["n"]
    return n, {"rmat": 1.9, "ba": 2.0}.get(case["graph"], 1.15) * case["deg"] * n


def work(case):
    nv, na = _sizes(case)
    csr, flops = 8.0 * nv + 4.0 * na, 0.0
    if case["kind"] == "train":
        flops = 3 * 2.0 * nv * sum(a * b for a, b in _WIDTHS)
        return dict(bytes=csr + 64.0 * nv + 2 * 4.0 * sum(a * b + b for a, b in _WIDTHS), flops=flops)
    if case["kind"] in ("propose", "learned"):
        flops = 2.0 * nv * sum(a * b for a, b in _WIDTHS)
    text = na * (1 + math.log10(max(10.0, nv))) if case["kind"] == "text" else 0.0
    labels = {"metrics": 4.0, "lp": 8.0}.get(case["kind"], 4.0) * nv
    return dict(bytes=csr + text + labels, flops=flops)


def exact(case, seed):
    """The training step in 64 bits (plain autograd; nothing is rounded to 16 bits).  The other kinds return
    whole numbers, and ratios of whole numbers."""
    if case["kind"] != "train":
        return None
    (vstart, off, col, _), X, y = _train_inputs(case, seed)
    vstart, off = torch.from_numpy(vstart).cuda(), torch.from_numpy(off).cuda()
    n = off.numel() - 1
    deg = off[1:] - off[:-1]
    size = vstart[1:] - vstart[:-1]
    inst = torch.repeat_interleave(torch.arange(size.numel(), device="cuda"), size)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    nbr = torch.from_numpy(col).cuda().long() + vstart[inst[row]]
    flat = torch.from_numpy(np.load(WEIGHTS)).cuda().double().requires_grad_()
    h, at = torch.from_numpy(X).cuda().double(), 0
    for i, (a, b) in enumerate(_WIDTHS):
        w, c = flat[at: at + a * b].view(a, b), flat[at + a * b: at + a * b + b]
        at += a * b + b
        mean = torch.zeros_like(h).index_add(0, row, h[nbr]) / deg.clamp(min=1)[:, None]
        h = torch.cat([h, mean], 1) @ w + c
        h = h.relu() if i < 2 else h
    score = torch.zeros(size.numel(), dtype=torch.float64, device="cuda").index_add(0, inst, h[:, 8]) / size
    loss = torch.nn.functional.binary_cross_entropy_with_logits(score, torch.from_numpy(y).cuda().double())
    (g,) = torch.autograd.grad(loss, flat)
    # Adam's first step from zero moments: both corrected moments are the gradient's own
    new = flat - _LR * g / (g.abs() + 1e-8)
    return dict(params=new.detach().cpu().numpy(), loss=float(loss))
