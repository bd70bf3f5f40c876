"""End-to-end training on the GPU through the drop-in Python API, compared
with the oracle's CPU training loop (community recall@10 within 1 point)."""
import numpy as np
import pytest

import cloverleaf_gb300 as cl
from cloverleaf_gb300 import _native, datagen
from tests._eval import community_recall

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sbm10k():
    return datagen.workload("sbm10k")


def gpu_learn(w, loss, form, seed=20222022, passes=None, valid_pct=0.0, **extra):
    ep = w["ep"]
    g = cl.Graph.from_csr(w["rows"], w["cols"], w["weights"])
    fs = cl.FeatureSet.from_csr(g, w["fptr"], w["fids"], w["n_feat"])
    lossobj = cl.EPLoss.starspace(ep["gamma"], ep["negatives"]) if loss == "starspace" else \
        cl.EPLoss.margin(ep["gamma"], ep["negatives"])
    prop = cl.EmbeddingPropagator(alpha=ep["alpha"], loss=lossobj, batch_size=ep["batch_size"], dims=ep["dims"],
                                  passes=passes or ep["passes"], seed=seed, max_nodes=ep["max_nodes"],
                                  valid_pct=valid_pct, indicator=False, form=form, **extra)
    emb = prop.learn_features(g, fs)
    return emb, prop.last_stats


def oracle_learn(oracle, w, loss):
    ep = w["ep"]
    table, st = oracle.train(w["rows"], w["cols"], w["weights"], w["fptr"], w["fids"], w["n_feat"], dims=ep["dims"],
                             alpha=ep["alpha"], loss=oracle.LOSS_STARSPACE if loss == "starspace" else
                             oracle.LOSS_MARGIN, gamma=ep["gamma"], negatives=ep["negatives"],
                             batch_size=ep["batch_size"], passes=ep["passes"],
                             max_nodes=(oracle.SAMPLE_FIXED, ep["max_nodes"]), threads=0)
    return table


@pytest.mark.parametrize("form", ["plain", "fused"])
@pytest.mark.parametrize("loss", ["starspace", "margin"])
def test_recall_matches_cpu_reference(oracle, sbm10k, loss, form):
    w = sbm10k
    emb, stats = gpu_learn(w, loss, form)
    assert emb.table.shape == (w["n_feat"], w["ep"]["dims"])
    assert np.isfinite(emb.table).all()
    assert len(stats) == w["ep"]["passes"]
    assert stats[-1]["train_loss"] < stats[0]["train_loss"]
    r_gpu = community_recall(w["fptr"], w["fids"], emb.table, w["community"])
    r_cpu = community_recall(w["fptr"], w["fids"], oracle_learn(oracle, w, loss), w["community"])
    assert abs(r_gpu - r_cpu) <= 0.01, (r_gpu, r_cpu)


def test_training_is_deterministic(sbm10k):
    a, _ = gpu_learn(sbm10k, "starspace", "fused", passes=2)
    b, _ = gpu_learn(sbm10k, "starspace", "fused", passes=2)
    assert np.array_equal(a.table, b.table)
    c, _ = gpu_learn(sbm10k, "starspace", "plain", passes=2)
    d, _ = gpu_learn(sbm10k, "starspace", "plain", passes=2)
    assert np.array_equal(c.table, d.table)


def test_pass_stats_and_validation(sbm10k):
    w = sbm10k
    emb, stats = gpu_learn(w, "starspace", "fused", passes=2, valid_pct=0.1)
    n_train = w["rows"].shape[0] - 1 - int(np.float32(10_000) * np.float32(0.1))
    for s in stats:
        assert s["anchors"] == n_train
        assert s["batches"] == -(-n_train // w["ep"]["batch_size"])
        assert 0 < s["kept_anchors"] <= s["anchors"]
        assert s["gathered_rows"] <= s["items"]
        assert 0 < s["unique_rows"] <= w["n_feat"] * s["batches"]
        assert s["alg_bytes"] > 0 and s["ms"] > 0
        assert np.isfinite(s["valid_loss"]) and s["valid_loss"] > 0


def test_drop_in_api_strings():
    # the reference's own usage: GraphBuilder + FeatureSet with string ids
    b = cl.GraphBuilder()
    rng = np.random.default_rng(0)
    for i in range(200):
        for j in rng.integers(0, 200, 3):
            if i != j:
                b.add_edge(("user", str(i)), ("user", str(int(j))), 1.0, cl.EdgeType.Undirected)
    g = b.build_graph()
    fs = cl.FeatureSet.new_from_graph(g)
    for i in range(0, 200, 2):   # odd nodes stay featureless
        fs.set_features(("user", str(i)), [("feat", f"t{i % 7}"), ("feat", f"t{i % 11}")])
    ep = cl.EmbeddingPropagator(alpha=0.05, loss=cl.EPLoss.starspace(0.5, 3), batch_size=32, dims=16, passes=3,
                                max_nodes=5, indicator=False)
    emb = ep.learn_features(g, fs)
    # fill_missing_nodes gave every odd node its own ("node", id) feature
    assert fs.get_features(("user", "1"))[0][0] == "node"
    assert emb.len() == fs.num_features() and emb.dims() == 16
    assert emb.contains(("feat", "t3"))
    nn = emb.nearest_neighbor(emb.get_embedding(("feat", "t3")), 3)
    assert nn[0][0] == ("feat", "t3")


def test_warm_start_moves_table_out(sbm10k):
    w = sbm10k
    emb, _ = gpu_learn(w, "starspace", "plain", passes=1)
    init = emb.table.copy()
    ep = w["ep"]
    g = cl.Graph.from_csr(w["rows"], w["cols"], w["weights"])
    fs = cl.FeatureSet.from_csr(g, w["fptr"], w["fids"], w["n_feat"])
    prop = cl.EmbeddingPropagator(alpha=ep["alpha"], loss=cl.EPLoss.starspace(0.5, 5), batch_size=256, dims=64,
                                  passes=1, max_nodes=10, valid_pct=0.0, indicator=False)
    out = prop.learn_features(g, fs, emb)
    assert emb.dims() == 0                 # moved out, as lib.rs:1337-1341
    assert out.table.shape == init.shape
    assert not np.array_equal(out.table, init)


def test_unsupported_options_raise():
    with pytest.raises(NotImplementedError):
        cl.EmbeddingPropagator(attention=8)
    with pytest.raises(ValueError):
        cl.EmbeddingPropagator(max_features=-1.0)


def test_large_chung_lu_batches():
    # 2% of the 10M-node workload: same degree and feature distributions
    w = datagen.workload("cl10m", scale=0.02)
    cfg = _native.default_config()
    ep = w["ep"]
    cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = ep["dims"], ep["negatives"], _native.LOSS_STARSPACE, ep["gamma"]
    cfg.batch_size, cfg.alpha, cfg.passes, cfg.valid_pct = 2048, ep["alpha"], 1, 0.0
    cfg.max_nodes_kind, cfg.max_nodes = _native.SAMPLE_FIXED, float(ep["max_nodes"])
    cfg.form = _native.FORM_FUSED_BF16
    ctx = _native.Context(cfg)
    ctx.upload_graph(w["rows"], w["cols"], None)
    ctx.upload_features(w["fptr"], w["fids"], w["n_feat"])
    ctx.set_table(None)
    s1 = ctx.train_batches(10)
    ctx.train_batches(150)
    s2 = ctx.train_batches(10)
    assert s1["kept_anchors"] > 0 and s1["nan_anchors"] == 0
    assert s2["train_loss"] < s1["train_loss"]
    t = ctx.get_table(w["n_feat"], ep["dims"])
    assert np.isfinite(t).all()


def _cl_ctx(w, form=_native.FORM_FUSED_BF16, autotune=0):
    return _cl_ctx_cfg(w, form=form, autotune=autotune)


def _cl_ctx_cfg(w, form=_native.FORM_FUSED_BF16, autotune=0, use_graphs=1):
    cfg = _native.default_config()
    cfg.use_graphs = use_graphs
    ep = w["ep"]
    cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = ep["dims"], ep["negatives"], _native.LOSS_STARSPACE, ep["gamma"]
    cfg.batch_size, cfg.alpha, cfg.passes, cfg.valid_pct = 2048, ep["alpha"], 1, 0.0
    cfg.max_nodes_kind, cfg.max_nodes = _native.SAMPLE_FIXED, float(ep["max_nodes"])
    cfg.form, cfg.autotune = form, autotune
    ctx = _native.Context(cfg)
    ctx.upload_graph(w["rows"], w["cols"], None)
    ctx.upload_features(w["fptr"], w["fids"], w["n_feat"])
    ctx.set_table(None)
    return ctx


def test_multi_batch_graph_matches_single_batch_graphs(monkeypatch):
    # runs of 16 batches replay one graph; the result must equal one graph
    # replay per batch bit for bit (same kernels, same order)
    w = datagen.workload("cl10m", scale=0.005)
    tables = []
    for gb in ("16", "1"):
        monkeypatch.setenv("EP_GRAPH_BATCHES", gb)
        ctx = _cl_ctx(w)
        assert ctx.tuning()[3] == int(gb)
        ctx.train_batches(37)
        tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert np.array_equal(tables[0], tables[1])


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
@pytest.mark.parametrize("ctas", ["1", "608"])
def test_persistent_reducer_gives_the_same_table(monkeypatch, form, ctas):
    # warps taking reducer chunks from a work counter (down to a single CTA)
    # reduce every chunk as the one-warp-per-chunk grid does
    w = datagen.workload("cl10m", scale=0.005)
    tables = []
    for r in ("0", ctas):
        monkeypatch.setenv("EP_RED_CTAS", r)
        ctx = _cl_ctx(w, form=form)
        st = ctx.train_batches(23)
        assert st["kept_anchors"] > 0
        tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert np.array_equal(tables[0], tables[1])


@pytest.mark.parametrize("warps", ["1", "2"])
def test_sampler_cta_size_gives_the_same_table(monkeypatch, warps):
    w = datagen.workload("cl10m", scale=0.005)
    tables = []
    for g in ("8", warps):
        monkeypatch.setenv("EP_SAMPLE_WARPS", g)
        ctx = _cl_ctx(w)
        ctx.train_batches(19)
        tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert np.array_equal(tables[0], tables[1])


@pytest.mark.parametrize("warps", ["1", "2", "4"])
def test_gather_cta_size_gives_the_same_table(monkeypatch, warps):
    w = datagen.workload("cl10m", scale=0.005)
    tables = []
    for g in ("8", warps):
        monkeypatch.setenv("EP_GATHER_WARPS", g)
        for graphs in (1, 0):
            ctx = _cl_ctx_cfg(w, use_graphs=graphs)
            ctx.train_batches(19)
            tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert all(np.array_equal(tables[0], t) for t in tables[1:])


def test_five_cta_queue_reducer_gives_the_same_table(monkeypatch):
    w = datagen.workload("cl10m", scale=0.005)
    tables = []
    for q in ("4", "5"):
        monkeypatch.setenv("EP_QUEUE_CTAS", q)
        ctx = _cl_ctx(w)
        assert ctx.launch_shape()["queue_ctas_per_sm"] == int(q)
        ctx.train_batches(29)
        tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert np.array_equal(tables[0], tables[1])


@pytest.mark.parametrize("mode", ["0", "1", "3"])
def test_adam_placements_give_the_same_table(monkeypatch, mode):
    # the fused form's Adam placements -- per row as each feature closes (0),
    # a separate kernel over dense gradient rows (1), the per-warp queue (2,
    # the reference point) and the warp-specialised ring with bulk copies (3)
    # -- apply the same update to the same reduced rows: equal tables, bit for bit
    w = datagen.workload("cl10m", scale=0.005)
    tables = []
    for m in ("2", mode):
        monkeypatch.setenv("EP_FUSED_MODE", m)
        ctx = _cl_ctx(w)
        assert ctx.tuning()[2] == int(m)
        st = ctx.train_batches(37)
        assert st["kept_anchors"] > 0
        tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert np.array_equal(tables[0], tables[1])


@pytest.mark.parametrize("ctas", ["1", "152", "608"])
def test_persistent_gather_gives_the_same_table(monkeypatch, ctas):
    # the staged gather as a persistent grid whose warps take anchors from a
    # work queue (any grid size, down to one CTA) computes every anchor as
    # the one-warp-per-anchor grid does
    w = datagen.workload("cl10m", scale=0.005)
    tables = []
    for g in ("0", ctas):
        monkeypatch.setenv("EP_GATHER_CTAS", g)
        for graphs in (1, 0):
            ctx = _cl_ctx_cfg(w, use_graphs=graphs)
            ctx.train_batches(19)
            tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert all(np.array_equal(tables[0], t) for t in tables[1:])


@pytest.mark.parametrize("shape", [("12", "4", "32"), ("6", "2", "4"), ("2", "14", "56"), ("1", "1", "2"),
                                   ("15", "1", "3")])
def test_ring_shapes_give_the_same_table(monkeypatch, shape):
    # reducing warps, Adam warps and slots per CTA of the ring change the
    # schedule only; tiny rings make every slot wrap many times
    w = datagen.workload("cl10m", scale=0.005)
    monkeypatch.setenv("EP_FUSED_MODE", "2")
    ref = _cl_ctx(w)
    ref.train_batches(21)
    want = ref.get_table(w["n_feat"], w["ep"]["dims"])
    monkeypatch.setenv("EP_FUSED_MODE", "3")
    for k, v in zip(("EP_RING_PW", "EP_RING_CW", "EP_RING_SLOTS"), shape):
        monkeypatch.setenv(k, v)
    ctx = _cl_ctx(w)
    ctx.train_batches(21)
    assert np.array_equal(ctx.get_table(w["n_feat"], w["ep"]["dims"]), want)


def test_graph_replays_match_stream_launches():
    # captured batches run k_batch_end on a side branch beside the sort and
    # reduction; the table and the pass statistics must equal those of the
    # same batches launched one kernel after another on one stream
    w = datagen.workload("cl10m", scale=0.005)
    out = []
    for graphs in (1, 0):
        ctx = _cl_ctx_cfg(w, use_graphs=graphs)
        st = ctx.train_batches(37)
        out.append((ctx.get_table(w["n_feat"], w["ep"]["dims"]), st))
    assert np.array_equal(out[0][0], out[1][0])
    same = ("pass", "batches", "train_loss", "lr_last", "anchors", "kept_anchors", "items", "gathered_rows",
            "unique_rows", "sampled_neighbors")
    assert {k: out[0][1][k] for k in same} == {k: out[1][1][k] for k in same}


def test_graph_replays_match_stream_launches_with_direct_gathers():
    # anchors too big for the staged gather's tables take the direct path,
    # in replayed graphs with their items from k_fwd_emit's direct walk
    from tests._cases import random_problem
    prob = random_problem(97, n=3000, n_feat=20000, dims=64, deg=(4, 30), feats=(10, 40))
    tables = []
    for graphs in (1, 0):
        cfg = _native.default_config()
        cfg.use_graphs = graphs
        cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = 64, 10, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.passes, cfg.valid_pct = 256, 1, 0.0
        cfg.max_nodes_kind, cfg.max_nodes = _native.SAMPLE_FIXED, 25.0
        ctx = _native.Context(cfg)
        ctx.upload_graph(prob["rows"], prob["cols"], None)
        ctx.upload_features(prob["fptr"], prob["fids"], prob["n_feat"])
        ctx.set_table(None)
        st = ctx.train_batches(20)
        assert st["kept_anchors"] > 0
        tables.append(ctx.get_table(prob["n_feat"], 64))
    assert np.array_equal(tables[0], tables[1])


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
@pytest.mark.parametrize("level", [1, 2])
def test_autotune_picks_a_candidate_and_trains(form, level):
    w = datagen.workload("cl10m", scale=0.01)
    ctx = _cl_ctx(w, form=form, autotune=level)
    assert ctx.tuning()[0] is False
    s1 = ctx.train_batches(260)          # the candidates' batches (200 at most), then more
    shape = ctx.launch_shape()
    tuned, chunk, mode, _ = ctx.tuning()
    assert tuned and shape["tuned"] and shape["autotune"] == level
    assert chunk == 128 if level == 1 else chunk in (64, 128, 256)
    if form == _native.FORM_FUSED_BF16:
        assert mode in ((2, 3) if level == 1 else (1, 2, 3))
    assert shape["gather_ctas"] in (0, 304, 456) and shape["gather_warps"] in (2, 4, 8)
    ctx.train_batches(120)
    s2 = ctx.train_batches(10)
    assert s2["train_loss"] < s1["train_loss"]
    assert np.isfinite(ctx.get_table(w["n_feat"], w["ep"]["dims"])).all()
    # a second context on the same workload starts with the remembered choice
    again = _cl_ctx(w, form=form, autotune=level)
    again.train_batches(1)
    assert again.launch_shape() == shape


def test_level_one_tuning_keeps_results_identical():
    # level 1 only chooses between launch shapes that give the same bits
    w = datagen.workload("cl10m", scale=0.01)
    tables = []
    for level in (0, 1):
        ctx = _cl_ctx(w, autotune=level)
        ctx.train_batches(110)
        tables.append(ctx.get_table(w["n_feat"], w["ep"]["dims"]))
    assert np.array_equal(tables[0], tables[1])


@pytest.mark.parametrize("max_features", [None, 3.0, 0.4])
def test_gather_split_gives_the_same_table(monkeypatch, max_features):
    # 1, 2 or 4 warps per anchor; nodes of 1 to 40 features (dropout packs
    # whole nodes of up to 32 into a step), some anchors past the tables
    from tests._cases import random_problem
    prob = random_problem(98, n=2000, n_feat=5000, dims=52, deg=(1, 30), feats=(1, 40))
    tables = []
    for split in ("1", "2", "4"):
        monkeypatch.setenv("EP_GATHER_SPLIT", split)
        for form, graphs in ((_native.FORM_FUSED_BF16, 1), (_native.FORM_FUSED_BF16, 0)):
            cfg = _native.default_config()
            cfg.use_graphs, cfg.form = graphs, form
            cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = 52, 7, _native.LOSS_STARSPACE, 0.5
            cfg.batch_size, cfg.passes, cfg.valid_pct = 300, 10, 0.0
            cfg.max_nodes_kind, cfg.max_nodes = _native.SAMPLE_FIXED, 20.0
            if max_features is not None:
                cfg.max_features = max_features
                cfg.max_features_kind = _native.SAMPLE_PROB if max_features < 1 else _native.SAMPLE_FIXED
            ctx = _native.Context(cfg)
            ctx.upload_graph(prob["rows"], prob["cols"], None)
            ctx.upload_features(prob["fptr"], prob["fids"], prob["n_feat"])
            ctx.set_table(None)
            assert ctx.train_batches(9)["kept_anchors"] > 0
            tables.append(ctx.get_table(prob["n_feat"], 52))
    assert all(np.array_equal(tables[0], t) for t in tables[1:])


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
@pytest.mark.parametrize("n_feat", [3, 40, 4000])
def test_reducer_split_gives_the_same_table(monkeypatch, form, n_feat):
    # 1, 2 or 4 warps per reducer chunk: chunks inside one hot feature (3
    # features), of a few features, and of one feature per item; the last
    # chunk ragged
    from tests._cases import random_problem
    prob = random_problem(99, n=1500, n_feat=n_feat, dims=36, deg=(1, 9), feats=(1, 5))
    tables = []
    for split in ("1", "2", "4"):
        monkeypatch.setenv("EP_RED_SPLIT", split)
        cfg = _native.default_config()
        cfg.form, cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = form, 36, 4, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.passes, cfg.valid_pct = 150, 1, 0.0
        ctx = _native.Context(cfg)
        ctx.upload_graph(prob["rows"], prob["cols"], None)
        ctx.upload_features(prob["fptr"], prob["fids"], prob["n_feat"])
        ctx.set_table(None)
        st = ctx.train_batches(7)
        assert st["kept_anchors"] > 0
        tables.append((ctx.get_table(prob["n_feat"], 36), st["unique_rows"], st["gathered_rows"]))
    for t, u, g in tables[1:]:
        assert np.array_equal(tables[0][0], t) and (u, g) == tables[0][1:]


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
@pytest.mark.parametrize("n_feat,batch", [(200, 7), (200, 400), (40_000, 130), (70_000, 500)])
def test_one_kernel_sort_passes_match_three(form, n_feat, batch):
    # small batches in replayed graphs sort by one kernel per pass, counted by
    # the item emission; stream launches by three.  1, 2 and 3 passes; less
    # than one tile of items, and several with a ragged last one
    from tests._cases import random_problem
    prob = random_problem(95, n=2000, n_feat=n_feat, dims=20, deg=(1, 20), feats=(1, 12))
    out = []
    for graphs in (1, 0):
        cfg = _native.default_config()
        cfg.use_graphs, cfg.form = graphs, form
        cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = 20, 3, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.passes, cfg.valid_pct = batch, 10, 0.0   # batches enough for replaying to pay
        ctx = _native.Context(cfg)
        ctx.upload_graph(prob["rows"], prob["cols"], None)
        ctx.upload_features(prob["fptr"], prob["fids"], n_feat)
        ctx.set_table(None)
        st = ctx.train_batches(11)
        out.append((ctx.get_table(n_feat, 20), st["kept_anchors"], st["items"], st["gathered_rows"], st["unique_rows"]))
    assert out[0][1] > 0 and out[0][1:] == out[1][1:] and np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
def test_one_kernel_sort_passes_only_where_no_batch_is_large(form):
    # the one-kernel passes do work in the square of a batch's items: a graph
    # whose typical batch is small, but where one hub's neighbourhood is not,
    # sorts by three kernels per pass (2 passes here), as the launch counts say
    def graph(hub):
        n = 250_000
        rows, cols = np.arange(n + 1, dtype=np.uint64), np.zeros(n, np.uint32)
        if hub:     # node 0 next to all others
            rows[1:] += n - 2
            cols = np.concatenate([np.arange(1, n), np.zeros(n - 1)]).astype(np.uint32)
        rng = np.random.default_rng(11)
        fptr = np.arange(n + 1, dtype=np.uint64) * 5
        return rows, cols, fptr, rng.integers(0, 40_000, 5 * n).astype(np.uint32)

    kernels, out = {}, []
    for hub, graphs in ((False, 1), (True, 1), (True, 0)):
        rows, cols, fptr, fids = graph(hub)
        cfg = _native.default_config()
        cfg.use_graphs, cfg.form = graphs, form
        cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = 16, 3, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.passes, cfg.valid_pct = 64, 1, 0.0
        ctx = _native.Context(cfg)
        ctx.upload_graph(rows, cols, None)
        ctx.upload_features(fptr, fids, 40_000)
        ctx.set_table(None)
        st = ctx.train_batches(16)
        assert st["kept_anchors"] > 0
        kernels[hub, graphs] = st["launches"] / 16
        if hub:
            out.append((ctx.get_table(40_000, 16), st["kept_anchors"], st["items"], st["unique_rows"]))
    # two more kernels in each pass, and the direct gather of anchors beyond the tables
    assert kernels[True, 1] - kernels[False, 1] == 2 * 2 + 1, kernels
    assert out[0][1:] == out[1][1:] and np.array_equal(out[0][0], out[1][0])


def _small_run(form, passes, graphs=1, steps=5):
    from tests._cases import random_problem
    prob = random_problem(94, n=steps * 60, n_feat=300, dims=16, deg=(1, 6), feats=(1, 4))
    cfg = _native.default_config()
    cfg.use_graphs, cfg.form = graphs, form
    cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = 16, 3, _native.LOSS_STARSPACE, 0.5
    cfg.batch_size, cfg.passes, cfg.valid_pct, cfg.autotune = 60, passes, 0.0, 0
    ctx = _native.Context(cfg)
    ctx.upload_graph(prob["rows"], prob["cols"], None)
    ctx.upload_features(prob["fptr"], prob["fids"], 300)
    ctx.set_table(None)
    return ctx


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
def test_long_runs_of_short_passes_are_replayed(form):
    # replayed batches have other kernels than launched ones (item emission,
    # one-kernel sort passes): the launch counts say which a run took
    replayed = _small_run(form, passes=100).train_batches(200)["launches"] / 200
    launched = _small_run(form, passes=100, graphs=0).train_batches(200)["launches"] / 200
    assert replayed != launched
    ctx = _small_run(form, passes=1)
    assert ctx.train_batches(5)["launches"] == 5 * launched      # as configured: too short to pay
    assert ctx.train_batches(300)["launches"] == 300 * replayed
    # as many batches one at a time: replayed once they have come to a run that pays
    one = _small_run(form, passes=1)
    per = [one.train_batches(1)["launches"] for _ in range(305)]
    assert per[0] == launched and per[-1] == replayed and per == sorted(per, key=lambda x: x == replayed)
    ref = _small_run(form, passes=1, graphs=0)
    ref.train_batches(305)
    want = ref.get_table(300, 16)
    assert np.array_equal(ctx.get_table(300, 16), want) and np.array_equal(one.get_table(300, 16), want)


def test_graph_size_follows_the_run(monkeypatch):
    # a run far past the configured passes takes graphs of several batches,
    # not one graph of the whole run
    ref = _small_run(_native.FORM_FUSED_BF16, passes=1, graphs=0, steps=5)
    ref.train_batches(5 + 500 + 17)
    want = ref.get_table(300, 16)
    ctx = _small_run(_native.FORM_FUSED_BF16, passes=1, steps=5)
    ctx.train_batches(5)
    assert ctx.launch_shape()["graph_batches"] == 1
    ctx.train_batches(500)
    assert 2 <= ctx.launch_shape()["graph_batches"] <= 16
    ctx.train_batches(17)
    assert np.array_equal(ctx.get_table(300, 16), want)
    # graphs of one batch: whole runs of up to 16, else batch by batch
    monkeypatch.setenv("EP_GRAPH_BATCHES", "1")
    one = _small_run(_native.FORM_FUSED_BF16, passes=1, steps=5)
    for n in (5, 1, 17, 499):
        one.train_batches(n)
    assert one.launch_shape()["graph_batches"] == 1
    assert np.array_equal(one.get_table(300, 16), want)


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
@pytest.mark.parametrize("batch", [1024, 1025, 1281, 2049, 3073, 4097])
def test_gather_split_by_batch_size_gives_the_same_table(monkeypatch, form, batch):
    # batch sizes on either side of each line of the rule, replayed (the sort
    # beside the gather) and launched
    from tests._cases import random_problem
    prob = random_problem(93, n=9000, n_feat=4000, dims=130, deg=(1, 12), feats=(1, 6))
    tables = []
    for split, graphs in ((None, 1), (None, 0), ("1", 1)):
        if split:
            monkeypatch.setenv("EP_GATHER_SPLIT", split)
        cfg = _native.default_config()
        cfg.use_graphs, cfg.form = graphs, form
        cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = 130, 5, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.passes, cfg.valid_pct, cfg.autotune = batch, 20, 0.0, 0
        ctx = _native.Context(cfg)
        ctx.upload_graph(prob["rows"], prob["cols"], None)
        ctx.upload_features(prob["fptr"], prob["fids"], 4000)
        ctx.set_table(None)
        assert ctx.train_batches(7)["kept_anchors"] > 0
        tables.append(ctx.get_table(4000, 130))
    assert all(np.array_equal(tables[0], t) for t in tables[1:])


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
@pytest.mark.parametrize("chunks,n_feat", [(1360, 50_000), (1376, 50_000), (3640, 50_000), (3660, 50_000), (905, 10_000),
                                           (920, 10_000), (1820, 50_000), (1830, 50_000), (600, 1190), (600, 1210), (600, 7)])
def test_reducer_split_by_chunk_count_gives_the_same_table(monkeypatch, form, chunks, n_feat):
    # batches on either side of each line of the rule (chunks of 128 items,
    # features per chunk): one feature a node, five nodes an anchor, so a batch
    # of b anchors emits 5 b items
    rng = np.random.default_rng(chunks)
    batch = chunks * 128 // 5
    n = 3 * batch
    rows = np.arange(n + 1, dtype=np.uint64)
    cols = rng.integers(0, n, n).astype(np.uint32)
    fids = rng.integers(0, n_feat, n).astype(np.uint32)
    out = []
    for split in (None, "1"):
        if split:
            monkeypatch.setenv("EP_RED_SPLIT", split)
        cfg = _native.default_config()
        cfg.form, cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = form, 36, 3, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.passes, cfg.valid_pct, cfg.autotune = batch, 20, 0.0, 0
        ctx = _native.Context(cfg)
        ctx.upload_graph(rows, cols, None)
        ctx.upload_features(rows, fids, n_feat)
        ctx.set_table(None)
        st = ctx.train_batches(4)
        assert st["kept_anchors"] > 0 and abs(st["items"] / 4 / 128 - chunks) < 2
        out.append((ctx.get_table(n_feat, 36), st["unique_rows"], st["gathered_rows"]))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]


@pytest.mark.parametrize("form,dims,batches", [(_native.FORM_FUSED_BF16, 256, 90), (_native.FORM_FUSED_BF16, 100, 70),
                                                (_native.FORM_PLAIN_FP32, 256, 50)])
def test_autotune_tries_no_shape_twice(form, dims, batches):
    # 1,000 anchors: several warps per chunk (no five-CTA reducer) and per
    # anchor (no CTA sizes of the one-warp gather); the shortest run that is
    # tuned stays that of all candidates, ten batches each
    w = datagen.workload("cl10m", scale=0.003)

    def context(level):
        cfg = _native.default_config()
        cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = dims, 10, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.alpha, cfg.passes, cfg.valid_pct = 1000, 0.01, 1, 0.0
        cfg.max_nodes_kind, cfg.max_nodes = _native.SAMPLE_FIXED, 25.0
        cfg.form, cfg.autotune = form, level
        ctx = _native.Context(cfg)
        ctx.upload_graph(w["rows"], w["cols"], None)
        ctx.upload_features(w["fptr"], w["fids"], w["n_feat"])
        ctx.set_table(None)
        return ctx

    ctx = context(1)
    ctx.train_batches(batches - 1)
    assert not ctx.launch_shape()["tuned"]
    ctx.train_batches(batches)
    shape = ctx.launch_shape()
    assert shape["tuned"] and shape["queue_ctas_per_sm"] == 4
    assert (shape["gather_ctas"], shape["gather_warps"]) in ((0, 2), (304, 8), (456, 8))
    ref = context(0)
    ref.train_batches(2 * batches - 1)
    assert np.array_equal(ctx.get_table(w["n_feat"], dims), ref.get_table(w["n_feat"], dims))


def _table_under(monkeypatch, env, make, batches):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    ctx, n_feat, dims = make()
    st = ctx.train_batches(batches)
    assert st["kept_anchors"] > 0
    for k in env:
        monkeypatch.delenv(k)
    return ctx.get_table(n_feat, dims)


@pytest.mark.parametrize("warps", ["1", "2", "4"])
@pytest.mark.parametrize("graphs", [1, 0])
def test_gather_cta_sizes_with_a_warp_per_anchor(monkeypatch, warps, graphs):
    # (batches of this size take several warps per anchor when left to the
    # rule, and the gather then has no CTA size)
    w = datagen.workload("cl10m", scale=0.005)
    make = lambda: (_cl_ctx_cfg(w, use_graphs=graphs), w["n_feat"], w["ep"]["dims"])  # noqa: E731
    tables = [_table_under(monkeypatch, {"EP_GATHER_SPLIT": "1", "EP_GATHER_WARPS": g}, make, 19) for g in ("8", warps)]
    assert np.array_equal(tables[0], tables[1])


def test_five_cta_reducer_with_a_warp_per_chunk(monkeypatch):
    # (batches of this size take several warps per chunk when left to the
    # rule, in a kernel of their own)
    w = datagen.workload("cl10m", scale=0.005)
    make = lambda: (_cl_ctx(w), w["n_feat"], w["ep"]["dims"])  # noqa: E731
    tables = [_table_under(monkeypatch, {"EP_RED_SPLIT": s, "EP_QUEUE_CTAS": q}, make, 29)
              for s, q in (("1", "4"), ("1", "5"), ("2", "4"))]
    assert np.array_equal(tables[0], tables[1]) and np.array_equal(tables[0], tables[2])


@pytest.mark.parametrize("chunk", ["128", "160", "512"])
@pytest.mark.parametrize("dims", [129, 130, 136, 200, 250, 255, 256])
def test_streamed_reducer_gives_the_queue_reducers_table(monkeypatch, dims, chunk):
    # BF16 rows of 129 to 256 dims: direction rows through the shared-memory
    # ring (a warp per chunk, four CTAs) against registers (five CTAs, or four
    # warps per chunk where a chunk is one window); lanes past the row, hot
    # features and chunks of a feature per item, a ragged last window
    from tests._cases import random_problem
    for n_feat in (5, 6000):
        prob = random_problem(dims, n=1500, n_feat=n_feat, dims=dims, deg=(1, 9), feats=(1, 5))

        def make():
            cfg = _native.default_config()
            cfg.form, cfg.dims, cfg.negatives = _native.FORM_FUSED_BF16, dims, 4
            cfg.loss, cfg.gamma, cfg.batch_size, cfg.passes, cfg.valid_pct = _native.LOSS_STARSPACE, 0.5, 400, 1, 0.0
            ctx = _native.Context(cfg)
            ctx.upload_graph(prob["rows"], prob["cols"], None)
            ctx.upload_features(prob["fptr"], prob["fids"], n_feat)
            ctx.set_table(None)
            return ctx, n_feat, dims

        shapes = [("1", "4"), ("1", "5")] + ([("4", "4")] if chunk == "128" else [])
        tables = [_table_under(monkeypatch, {"EP_REDUCE_CHUNK": chunk, "EP_RED_SPLIT": s, "EP_QUEUE_CTAS": q}, make, 7)
                  for s, q in shapes]
        assert all(np.array_equal(tables[0], t) for t in tables[1:])


@pytest.mark.parametrize("form", [_native.FORM_FUSED_BF16, _native.FORM_PLAIN_FP32])
def test_training_again_on_a_context_equals_a_new_one(form):
    # a new table leaves the captured graphs in place: the second and third
    # runs replay them, after a given table as after a drawn one, after another
    # run length and after explicit batches that grow the scratch
    from tests._cases import random_problem, sample_batch
    prob = random_problem(92, n=3000, n_feat=2000, dims=40, deg=(1, 9), feats=(1, 5))
    small = sample_batch(1, prob, B=50, K=6, R=4)
    large = sample_batch(2, prob, B=900, K=9, R=4)

    def context():
        cfg = _native.default_config()
        cfg.form, cfg.dims, cfg.negatives, cfg.loss, cfg.gamma = form, 40, 4, _native.LOSS_STARSPACE, 0.5
        cfg.batch_size, cfg.passes, cfg.valid_pct, cfg.autotune = 100, 2, 0.1, 0
        ctx = _native.Context(cfg)
        ctx.upload_graph(prob["rows"], prob["cols"], None)
        ctx.upload_features(prob["fptr"], prob["fids"], 2000)
        return ctx

    def run(ctx, table, batches):
        ctx.set_table(table)
        stats = ctx.train_batches(batches) if batches else ctx.train(2)[-1]
        same = ("train_loss", "valid_loss", "lr_last", "kept_anchors", "items", "gathered_rows", "unique_rows")
        return ctx.get_table(2000, 40), [stats[k] for k in same]

    used = context()
    for table, batches, between in ((None, 0, None), (prob["table"], 0, small), (None, 45, large), (prob["table"], 7, None),
                                    (None, 0, small), (None, 45, None)):
        got, want = run(used, table, batches), run(context(), table, batches)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1], equal_nan=True)
        if between:
            used.batch_grad(_native.Context.samples(between["anchors"], between["nbr_ptr"], between["nbr"], between["nbr_w"],
                                                    between["neg"]), 2000, 40)
