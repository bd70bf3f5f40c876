"""The framework's work as a user's program calls it: training from scratch
(EmbeddingPropagator.learn_features), retraining on an uploaded graph
(Context.train), the differentiable batch loss (EPBatchLoss), and the
evaluation calls on host arrays (node embeddings, cosine neighbours,
neighbourhood alignment).  Sizes follow the named workloads of
cloverleaf_gb300/datagen.py, with fewer nodes where a pass would take long:
batch size, dims, neighbour and negative counts and feature distributions are
theirs.

listed() the cases; draw(rng) one more of the same ranges; prepare(case, seed)
what the program holds before the call; run(state) one pass; work(case) the
bytes and operations it cannot do without; exact(case, seed) the result in 64
bits where one exists.
"""
import math

import numpy as np
import torch

import cloverleaf_gb300 as cl
from cloverleaf_gb300 import _native, datagen, evaluate
from cloverleaf_gb300.autograd import EPBatchLoss

DEV = "cuda"


def listed():
    return [
        # The smallest call: a first try on a small graph with every option
        # left at the API's default (dims 100, batches of 50, one negative,
        # all neighbours, 10% validation nodes).
        _train("learn_defaults_2k", "learn", "sbm", 2_000, dims=100, batch=50, negatives=1, max_nodes=0, loss="margin",
               gamma=1.0, alpha=0.9, passes=1, valid=0.1),
        # The planted-community workload (sbm10k), whole call: context, upload,
        # two passes with validation, download.
        _train("learn_sbm10k", "learn", "sbm", 10_000, dims=64, batch=256, negatives=5, max_nodes=10, passes=2, valid=0.1),
        # The options used together on an odd width: margin loss, edge-weighted
        # sampling and averaging, feature dropout, hard negatives, log weighting.
        _train("train_options_d100_fused", "train", "cl1m", 60_000, slots=30_000, form="fused", dims=100, batch=1000,
               negatives=6, max_nodes=12, loss="margin", weighted=True, max_features=6, hard=2, log_weight=True),
        # The bipartite weighted workload (cl1m) in the plain form: batches of 1024.
        _train("train_cl1m_plain", "train", "cl1m", 200_000, slots=100_000, dims=128, batch=1024, negatives=10, max_nodes=25),
        # The 10M-node workload's batch (the benchmark's step), fused and plain.
        _train("train_cl10m_fused", "train", "cl10m", 500_000, slots=500_000, form="fused", dims=256, batch=8192,
               negatives=10, max_nodes=25),
        _train("train_cl10m_plain", "train", "cl10m", 500_000, slots=500_000, dims=256, batch=8192, negatives=10, max_nodes=25),
        # The 50M-node workload's batch: the largest training step.
        _train("train_cl50m_fused", "train", "cl50m", 1_000_000, slots=1_000_000, form="fused", dims=256, batch=32768,
               negatives=16, max_nodes=32),
        # The differentiable batch loss, forward and backward: the
        # differentiation-check workload (sbm1k) and a training-sized batch.
        _auto("autograd_sbm1k", 1_000, n_feat=2_500, dims=32, batch=128, negatives=5, k=10),
        _auto("autograd_b4096_d128", 100_000, n_feat=50_000, dims=128, batch=4096, negatives=10, k=25),
        # After training: node embeddings of a graph, its nearest neighbours
        # (a block of queries as the recall evaluation makes), and alignment.
        {"name": "embed_200k_d256", "kind": "embed", "nodes": 200_000, "slots": 100_000, "dims": 256},
        {"name": "knn_8192x262144_d256", "kind": "knn", "rows": 262_144, "queries": 8_192, "dims": 256, "k": 10},
        {"name": "align_200k_d128", "kind": "align", "nodes": 200_000, "dims": 128, "max_neighbors": 0, "alpha": 0.5},
    ]


def _train(name, kind, graph, nodes, *, slots=0, form="plain", dims, batch, negatives, max_nodes, loss="starspace",
           gamma=0.5, alpha=0.01, passes=1, valid=0.0, weighted=False, max_features=0, hard=0, log_weight=False):
    """graph: sbm, or the Chung-Lu family of cl1m / cl10m / cl50m; max_nodes and max_features 0 = all."""
    return {"name": name, "kind": kind, "graph": graph, "nodes": nodes, "slots": slots, "form": form, "dims": dims,
            "batch": batch, "negatives": negatives, "max_nodes": max_nodes, "loss": loss, "gamma": gamma, "alpha": alpha,
            "passes": passes, "valid": valid, "weighted": weighted, "max_features": max_features, "hard": hard,
            "log_weight": log_weight}


def _auto(name, nodes, *, n_feat, dims, batch, negatives, k, loss="starspace", double=False):
    return {"name": name, "kind": "autograd", "nodes": nodes, "n_feat": n_feat, "dims": dims, "batch": batch,
            "negatives": negatives, "k": k, "loss": loss, "double": double}


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choices(["learn", "train", "autograd", "embed", "knn", "align"], [3, 8, 3, 2, 2, 2])[0]
    if kind in ("learn", "train"):
        graph = "sbm" if kind == "learn" else rng.choice(["cl1m", "cl1m", "cl10m", "cl50m"])
        nodes = log_int(1_000, 20_000) if kind == "learn" else log_int(30_000, 500_000)
        dims = log_int(16, 256)
        # no more than about 200 batches a pass, and batches of up to 16384 anchors
        batch = log_int(max(32, nodes // 200), max(64, min(nodes // 4, 16_384)))
        c = _train("", kind, graph, nodes, slots=log_int(5_000, 500_000), form=rng.choice(["plain", "fused"]), dims=dims,
                   batch=batch, negatives=log_int(1, 16),
                   max_nodes=rng.choice([0, 10]) if graph == "sbm" else log_int(2, 32),
                   loss=rng.choice(["starspace", "starspace", "margin", "contrastive"]), valid=rng.choice([0.0, 0.1]))
        if graph == "cl1m":
            c["weighted"] = rng.random() < 0.3
        c["max_features"] = rng.choice([0, 0, 0, 4])
        c["log_weight"] = rng.random() < 0.2
        c["hard"] = min(c["negatives"], 2) if rng.random() < 0.15 else 0
    elif kind == "autograd":
        nodes = log_int(1_000, 100_000)
        c = _auto("", nodes, n_feat=log_int(1_000, 50_000), dims=log_int(16, 256), batch=log_int(64, 4_096),
                  negatives=log_int(1, 16), k=log_int(2, 25), loss=rng.choice(["starspace", "margin"]),
                  double=rng.random() < 0.25)
    elif kind == "embed":
        c = {"kind": "embed", "nodes": log_int(2_000, 300_000), "slots": log_int(2_000, 200_000), "dims": log_int(16, 256)}
    elif kind == "knn":
        c = {"kind": "knn", "rows": log_int(2_000, 300_000), "queries": log_int(16, 10_000), "dims": log_int(16, 256),
             "k": rng.choice([1, 5, 10, 20, 32])}
    else:
        c = {"kind": "align", "nodes": log_int(2_000, 300_000), "dims": log_int(16, 256),
             "max_neighbors": rng.choice([0, 0, 8]), "alpha": rng.choice([-1.0, 0.5, 0.8])}
    c.pop("name", None)
    return c


# nodes' features: (Poisson rate, fewest, most, Zipf exponent); mean degree
_FAMILY = {
    "cl1m": dict(exponent=2.1, mean_degree=20.0, max_degree=1e9, bipartite=True, w_hi=5.0, feat=(0.0, 1, 16, 1.1)),
    "cl10m": dict(exponent=2.0, mean_degree=16.0, max_degree=1e4, bipartite=False, w_hi=1.0, feat=(6.0, 1, 32, 1.05)),
    "cl50m": dict(exponent=2.1, mean_degree=20.0, max_degree=1e5, bipartite=False, w_hi=1.0, feat=(8.0, 1, 64, 1.1)),
}


def _graph(family, nodes, slots, seed):
    """Host CSR arrays (rows, cols, weights, fptr, fids, n_feat) of one workload family."""
    if family == "sbm":
        blocks = max(2, min(32, nodes // 100))
        rows, cols, w, comm = datagen.sbm(nodes, blocks, 8.0, 2.0, seed)
        fptr, fids, n_feat, _ = datagen.sbm_tokens(comm, 4, 8, 256, 8192, 0.8, 16, seed + 1)
        # the whole vocabulary has rows, whether or not a token turns up
        return rows, cols, w, fptr, fids, max(n_feat, 256 * blocks + 8192)
    g = _FAMILY[family]
    rows, cols, w = datagen.chung_lu(nodes, g["exponent"], g["mean_degree"], g["max_degree"], g["bipartite"], 1.0, g["w_hi"],
                                     seed)
    lam, lo, hi, s = g["feat"]
    fptr, fids = datagen.zipf_features(nodes, lam, lo, hi, s, slots, seed + 1)
    return rows, cols, w, fptr, fids, slots


def _propagator(c, seed):
    loss = {"margin": lambda: cl.EPLoss.margin(c["gamma"], c["negatives"]),
            "starspace": lambda: cl.EPLoss.starspace(c["gamma"], c["negatives"]),
            "contrastive": lambda: cl.EPLoss.contrastive(c["gamma"], 0.2, c["negatives"])}[c["loss"]]()
    return cl.EmbeddingPropagator(
        alpha=c["alpha"], loss=loss, batch_size=c["batch"], dims=c["dims"], passes=c["passes"], seed=seed,
        max_nodes=c["max_nodes"] or None, weighted_neighbor_sampling=c["weighted"],
        weighted_neighbor_averaging=c["weighted"], max_features=c["max_features"] or None,
        loss_weighting=cl.LossWeighting.Log() if c["log_weight"] else None, valid_pct=c["valid"],
        hard_negatives=c["hard"], indicator=False, form=c["form"])


def _samples(c, seed):
    """A graph, its features and one batch of explicit samples for the differentiable loss (numpy, CSR)."""
    rng = np.random.default_rng(seed)
    n, B, R, K = c["nodes"], c["batch"], c["negatives"], c["k"]
    deg = rng.integers(1, 25, n)
    rows = np.zeros(n + 1, np.uint64)
    rows[1:] = np.cumsum(deg)
    src = np.repeat(np.arange(n), deg)
    cols = rng.integers(0, n, int(rows[-1]))
    cols = np.where(cols == src, (cols + 1) % n, cols).astype(np.uint32)      # no loops
    cnt = rng.integers(2, 7, n)
    fptr = np.zeros(n + 1, np.uint64)
    fptr[1:] = np.cumsum(cnt)
    fids = (c["n_feat"] * rng.random(int(fptr[-1])) ** 2).astype(np.uint32)   # low ids are common
    anchors = rng.integers(0, n, B, dtype=np.uint32)
    take = np.minimum(deg[anchors], K)
    nbr_ptr = np.zeros(B + 1, np.uint32)
    nbr_ptr[1:] = np.cumsum(take)
    own = np.repeat(np.arange(B), take)
    within = np.arange(int(nbr_ptr[-1])) - np.repeat(nbr_ptr[:-1].astype(np.int64), take)
    start = rng.integers(0, deg[anchors])                                     # a run of the row's edges, cyclic
    pos = (start[own] + within) % deg[anchors][own]
    nbr = cols[rows[anchors[own]].astype(np.int64) + pos]
    nbr_w = (deg[anchors] / take).astype(np.float32)[own]
    neg = rng.integers(0, n, (B, R), dtype=np.uint32)
    # a negative that is the anchor's only neighbour has no direction from it (margin loss)
    neg = np.where(neg == nbr[nbr_ptr[:-1]][:, None], (neg + 1) % np.uint32(n), neg).astype(np.uint32)
    return dict(rows=rows, cols=cols, fptr=fptr, fids=fids, anchors=anchors, nbr_ptr=nbr_ptr, nbr=nbr, nbr_w=nbr_w, neg=neg)


def _rows(n, dims, seed, clusters=0):
    """Embedding rows as a host array: normal, around `clusters` centres if given."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(n, dims, generator=g, device=DEV)
    if clusters:
        centre = torch.randn(clusters, dims, generator=g, device=DEV)
        x = x * 0.7 + centre[torch.randint(0, clusters, (n,), generator=g, device=DEV)]
    return x.cpu().numpy()


def _loss_of(c):
    return cl.EPLoss.starspace(0.5, c["negatives"]) if c["loss"] == "starspace" else cl.EPLoss.margin(1.0, c["negatives"])


def prepare(case, seed):
    c = case
    if c["kind"] in ("learn", "train"):
        rows, cols, w, fptr, fids, n_feat = _graph(c["graph"], c["nodes"], c["slots"], seed)
        graph = cl.Graph.from_csr(rows, cols, w)
        feats = cl.FeatureSet.from_csr(graph, fptr, fids, n_feat)
        p = _propagator(c, seed)
        if c["kind"] == "learn":
            return {"case": c, "p": p, "graph": graph, "feats": feats}
        # the graph stays on the device; the result goes to page-locked memory
        out = torch.empty(n_feat, c["dims"], pin_memory=True)
        return {"case": c, "ctx": p.context(graph, feats), "n_feat": n_feat, "out": out}
    if c["kind"] == "autograd":
        s = _samples(c, seed)
        g = torch.Generator(device=DEV).manual_seed(seed)
        dt = torch.float64 if c["double"] else torch.float32
        table = (torch.randn(c["n_feat"], c["dims"], generator=g, device=DEV, dtype=dt) / 4).requires_grad_()
        f = EPBatchLoss(s["rows"], s["cols"], s["fptr"], s["fids"], c["n_feat"], c["dims"], _loss_of(c))
        return {"case": c, "f": f, "table": table, "args": (s["anchors"], s["nbr_ptr"], s["nbr"], s["nbr_w"], s["neg"])}
    if c["kind"] == "embed":
        fptr, fids = datagen.zipf_features(c["nodes"], 6.0, 1, 32, 1.05, c["slots"], seed)
        return {"case": c, "fptr": fptr, "fids": fids, "table": _rows(c["slots"], c["dims"], seed)}
    if c["kind"] == "knn":
        emb = _rows(c["rows"], c["dims"], seed, clusters=64)
        q = np.random.default_rng(seed).integers(0, c["rows"], c["queries"])
        store = cl.NodeEmbeddings(cl.Vocab.anonymous(c["rows"]), emb, cl.Distance.Cosine)
        return {"case": c, "store": store, "queries": emb[q], "self": q.astype(np.uint64)}
    rows, cols, w = datagen.chung_lu(c["nodes"], 2.1, 20.0, 1e4, False, 1.0, 5.0, seed)
    graph = cl.Graph.from_csr(rows, cols, w)
    store = cl.NodeEmbeddings(graph.vocab_, _rows(c["nodes"], c["dims"], seed), cl.Distance.Cosine)
    aligner = cl.NeighborhoodAligner(None if c["alpha"] < 0 else c["alpha"], c["max_neighbors"] or None)
    return {"case": c, "graph": graph, "store": store, "aligner": aligner}


def _stats(passes):
    """The counts and losses that training reports for each pass."""
    counts = ("batches", "anchors", "kept_anchors", "nan_anchors", "items", "gathered_rows", "unique_rows", "sampled_neighbors")
    return {"counts": np.array([[s[k] for k in counts] for s in passes], np.int64),
            "losses": np.array([[s["train_loss"], s["valid_loss"]] for s in passes], np.float32)}


def run(state):
    c = state["case"]
    if c["kind"] == "learn":
        emb = state["p"].learn_features(state["graph"], state["feats"])
        return {"table": emb.table, **_stats(state["p"].last_stats)}
    if c["kind"] == "train":
        ctx = state["ctx"]
        ctx.set_table(None)
        stats = ctx.train(c["passes"])
        return {"table": ctx.get_table(state["n_feat"], c["dims"], state["out"].numpy()), **_stats(stats)}
    if c["kind"] == "autograd":
        table = state["table"]
        table.grad = None
        loss = state["f"](table, *state["args"])
        loss.sum().backward()
        return {"loss": loss.detach(), "grad": table.grad}
    if c["kind"] == "embed":
        return evaluate.node_embeddings(state["fptr"], state["fids"], state["table"])
    if c["kind"] == "knn":
        ids, dist = state["store"].nearest_neighbors(state["queries"], c["k"], state["self"])
        return {"ids": ids, "dist": dist}
    return state["aligner"].align(state["store"], state["graph"]).table


def _distinct(draws, slots, s):
    """Expected number of different values in `draws` Zipf(s) draws from `slots`."""
    p = np.arange(1, slots + 1, dtype=np.float64) ** -s
    return float(-np.expm1(draws * np.log1p(-np.minimum(p / p.sum(), 1 - 1e-12))).sum())


def work(case):
    c = case
    d = c["dims"]
    if c["kind"] in ("learn", "train"):
        # each batch reads and writes the distinct rows it touches once (table
        # row, two FP32 moments) and the feature ids of its sampled nodes; a
        # pass starts from a new table and ends with its download
        sbm = c["graph"] == "sbm"
        lam, lo, hi, s = (0.0, 4, 8, 0.5) if sbm else _FAMILY[c["graph"]]["feat"]
        per_node = (lo + hi) / 2 if lam == 0 else lam
        if c["max_features"]:
            per_node = min(per_node, c["max_features"])
        deg = 10.0 if sbm else 0.4 * _FAMILY[c["graph"]]["mean_degree"]      # of a typical node
        sampled = min(deg, c["max_nodes"] or deg)
        slots = 14_000 if sbm else c["slots"]
        es = 2 if c["form"] == "fused" else 4
        nodes = c["batch"] * (1 + sampled + c["negatives"])
        items = nodes * per_node
        batches = c["passes"] * math.ceil(c["nodes"] * (1 - c["valid"]) / c["batch"])
        rows = _distinct(items, slots, s)
        upload = c["nodes"] * (16 + (10 if sbm else 20) * 8 + per_node * 4) if c["kind"] == "learn" else 0
        return {"bytes": batches * (rows * d * (2 * es + 16) + items * 4 + nodes * 16) + slots * d * (es + 8 + es + 4) + upload,
                "flops": batches * (4.0 * items * d + 20.0 * rows * d)}
    if c["kind"] == "autograd":
        items = c["batch"] * (1 + min(c["k"], 12) + c["negatives"]) * 4.0
        es = 8 if c["double"] else 4
        rows = c["n_feat"] * -math.expm1(-items / c["n_feat"])
        # the rows that are touched, the dense gradient, the samples
        return {"bytes": rows * d * es + c["n_feat"] * d * es + items * 4, "flops": 6.0 * items * d}
    if c["kind"] == "embed":
        return {"bytes": 4.0 * d * (c["nodes"] + c["slots"]) + c["nodes"] * (8 + 24), "flops": 6.0 * c["nodes"] * d}
    if c["kind"] == "knn":
        return {"bytes": 4.0 * d * (c["rows"] + c["queries"]) + 8.0 * c["queries"] * c["k"],
                "flops": 2.0 * c["rows"] * c["queries"] * d}
    deg = min(20, c["max_neighbors"] or 20)
    return {"bytes": 8.0 * d * c["nodes"] + c["nodes"] * (8 + 8 * 20), "flops": 2.0 * c["nodes"] * (deg + 1) * d}


def _seg(ptr):
    """Row of each entry of a CSR."""
    ptr = torch.as_tensor(ptr.astype(np.int64), device=DEV)
    return torch.repeat_interleave(torch.arange(len(ptr) - 1, device=DEV), ptr[1:] - ptr[:-1])


def exact(case, seed):
    c = case
    if c["kind"] in ("learn", "train"):
        return None     # the samples are the framework's own random draws
    if c["kind"] == "autograd":
        return _exact_autograd(c, seed)
    s = prepare(c, seed)
    if c["kind"] == "embed":
        seg, f = _seg(s["fptr"]), torch.as_tensor(s["fids"].astype(np.int64), device=DEV)
        table = torch.as_tensor(s["table"], device=DEV).double()
        out = torch.zeros(c["nodes"], c["dims"], dtype=torch.float64, device=DEV).index_add_(0, seg, table[f])
        return out / torch.bincount(seg, minlength=c["nodes"])[:, None]
    if c["kind"] == "knn":
        x = torch.as_tensor(s["store"].table, device=DEV).double()
        x = x / x.norm(dim=1, keepdim=True)
        own = torch.as_tensor(s["self"].astype(np.int64), device=DEV)
        best = []
        for b in range(0, len(own), 512):
            sim = x[own[b:b + 512]] @ x.T
            sim[torch.arange(len(sim), device=DEV), own[b:b + 512]] = -2
            best.append(1 - sim.topk(c["k"], dim=1).values)
        return {"ids": None, "dist": torch.cat(best)}
    rows, cols = s["graph"].rows.astype(np.int64), s["graph"].cols.astype(np.int64)
    deg = np.diff(rows)
    seg = _seg(s["graph"].rows)
    cdf = torch.as_tensor(s["graph"].weights, device=DEV).double()
    at = torch.arange(len(cols), device=DEV) - torch.as_tensor(rows[:-1], device=DEV)[seg]
    p = cdf - torch.where(at > 0, torch.cat([cdf.new_zeros(1), cdf[:-1]]), cdf.new_zeros(()))
    if c["max_neighbors"]:
        p = p * (at < c["max_neighbors"])
    x = torch.as_tensor(s["store"].table, device=DEV).double()
    near = torch.zeros_like(x)
    cols = torch.as_tensor(cols, device=DEV)
    for b in range(0, len(cols), 1 << 21):
        e = slice(b, b + (1 << 21))
        near.index_add_(0, seg[e], p[e, None] * x[cols[e]])
    d = torch.as_tensor(deg, device=DEV).double()
    a = torch.full_like(d, c["alpha"]) if c["alpha"] >= 0 else (1 / torch.log(d + 1)).clamp(max=1)
    return (1 - a)[:, None] * near + a[:, None] * x


def _exact_autograd(c, seed):
    """The batch loss and its gradient through torch's own autograd in 64 bits."""
    s = _samples(c, seed)
    g = torch.Generator(device=DEV).manual_seed(seed)
    dt = torch.float64 if c["double"] else torch.float32
    table = (torch.randn(c["n_feat"], c["dims"], generator=g, device=DEV, dtype=dt) / 4).double().requires_grad_()
    B, R = c["batch"], c["negatives"]
    fptr = torch.as_tensor(s["fptr"].astype(np.int64), device=DEV)
    fids = torch.as_tensor(s["fids"].astype(np.int64), device=DEV)

    def mean(nodes, role, weight, roles):
        """Mean feature row of each role over its nodes' features, a node's features weighing weight + 1."""
        n = fptr[nodes + 1] - fptr[nodes]
        own = torch.repeat_interleave(torch.arange(len(nodes), device=DEV), n)
        at = torch.arange(len(own), device=DEV) - torch.repeat_interleave(n.cumsum(0) - n, n)
        f, w, r = fids[fptr[nodes][own] + at], (weight + 1)[own], role[own]
        num = torch.zeros(roles, c["dims"], dtype=torch.float64, device=DEV).index_add(0, r, w[:, None] * table[f])
        return num / torch.zeros(roles, dtype=torch.float64, device=DEV).index_add(0, r, w)[:, None]

    one = lambda n: torch.ones(n, dtype=torch.float64, device=DEV)  # noqa: E731
    t = lambda a: torch.as_tensor(a.astype(np.int64), device=DEV)  # noqa: E731
    h = mean(t(s["anchors"]), torch.arange(B, device=DEV), one(B), B)
    near = mean(t(s["nbr"]), _seg(s["nbr_ptr"]), torch.as_tensor(s["nbr_w"], device=DEV).double(), B)
    u = mean(t(s["neg"].reshape(-1)), torch.arange(B * R, device=DEV), one(B * R), B * R).reshape(B, R, -1)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)  # noqa: E731
    if c["loss"] == "starspace":
        terms = 0.5 - ((unit(near) * unit(h)).sum(-1)[:, None] - (unit(h)[:, None] * unit(u)).sum(-1))
    else:
        terms = 1.0 + (near - h).norm(dim=-1)[:, None] - (near[:, None] - u).norm(dim=-1)
    kept = terms > 0
    loss = torch.where(kept, terms, torch.zeros_like(terms)).sum(1) / kept.sum(1).clamp(min=1)
    loss.sum().backward()
    return {"loss": loss.detach(), "grad": table.grad}
