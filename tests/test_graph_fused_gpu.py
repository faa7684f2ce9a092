"""GPU parity of the kernel that keeps whole graphs in shared memory across the levels (graph_fused.cu) with a float64
restatement of the classifier (kernel_mean_field.cpp:28-47), at the sizes where it can go wrong: graphs at the edges of a
row block and of the largest tile, empty and isolated ones, rows longer than the column list, equal and mixed edge
weights, dense inputs, one launch and several."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from conftest import assert_close
from graphnn_b200 import capi, engine, synth

pytestmark = pytest.mark.gpu


def make(sizes, degree, d, tags, levels, hidden, classes, seed):
    rng = np.random.default_rng(seed)
    sizes = np.asarray(sizes, np.int64)
    off = np.concatenate([[0], np.cumsum(sizes)])
    us, vs = [], []
    for g, n in enumerate(sizes):
        if n < 2:
            continue
        m = int(degree * n) if degree < n else n * n
        us.append(rng.integers(0, n, m) + off[g])      # duplicates and self loops kept
        vs.append(rng.integers(0, n, m) + off[g])
    src = np.concatenate(us).astype(np.int32) if us else np.zeros(0, np.int32)
    dst = np.concatenate(vs).astype(np.int32) if vs else np.zeros(0, np.int32)
    w = synth._weights(rng, tags, d, hidden, classes, 0.3 / np.sqrt(d * max(degree, 1)))
    return synth.GraphBatch(sizes.astype(np.int32), src, dst, rng.integers(0, tags, off[-1]).astype(np.int32), tags, d, levels, hidden,
                            classes, w, "custom")


def f64(b, rp, ci, val, x, average):
    w = {k: v.astype(np.float64) for k, v in b.weights.items()}
    N = b.num_nodes
    A = sp.csr_matrix((np.ones(len(ci)) if val is None else val.astype(np.float64), ci, rp), shape=(N, N))
    msg = (x.astype(np.float64) @ w["w_n2l"]) if x is not None else w["w_n2l"][b.tags]
    H = np.maximum(msg, 0)
    for _ in range(b.levels):
        H = np.maximum((A @ H) @ w["p_node_conv"] + msg, 0)
    off = b.graph_offsets()
    Y = np.stack([H[off[g]:off[g + 1]].sum(0) / (max(off[g + 1] - off[g], 1) if average else 1) for g in range(b.num_graphs)])
    return H, np.maximum(Y @ w["h1_weight"], 0) @ w["h2_weight"]


@pytest.mark.parametrize("d,sizes,degree,opts", [
    (64, [1, 2, 0, 127, 128, 5, 3], 2.0, {}),                       # one row block per tile
    (32, [1, 2, 0, 127, 128, 5, 3], 2.0, {"dense": True}),
    (128, [1, 2, 0, 127, 128, 5, 3], 2.0, {"auto": True}),
    (64, [129, 640, 0, 1, 255, 256, 257, 639], 6.5, {}),            # several row blocks, the largest graph
    (64, [640, 620, 100, 7], 6.5, {"val": "row", "average": True}),  # averaged messages
    (64, [300, 20], 6.5, {"val": "mixed"}),                         # weights that differ inside a row
    (64, [200, 100, 150], 60.0, {}),                                # more columns than the list holds
    (32, [1024, 641, 1000, 2], 5.0, {}),                            # d = 32 with 1,024-row tiles
    (32, [640, 130, 1, 300], 3.0, {"val": "row"}),
    (64, [20] * 700, 2.2, {"dense": True, "average": True}),        # several tiles per CTA
    (128, [1, 2, 0, 127, 128, 5, 3, 70], 2.0, {"auto": True, "dense": True}),          # dense rows at d = 128: one launch after the projection,
    (128, [50, 77, 128, 1] * 180, 2.2, {"dense": True, "average": True}),              # and several tiles per CTA
    (64, [3] * 3000, 1.0, {"auto": True}),                          # 64 graphs end a tile; the readout inside the kernel
    (128, [30] * 900, 2.2, {"auto": True, "average": True, "val": "row"}),
], ids=lambda v: None)
def test_fused_forward(d, sizes, degree, opts):
    b = make(sizes, degree, d, 9, 3, 128 if d != 32 else 64, 3, seed=d + len(sizes))
    rng = np.random.default_rng(7)
    eng = engine.S2VInference(b.weights, b.levels, pool_average=opts.get("average", False))
    if not opts.get("auto"):
        eng.ctx.set_option(eng.ctx.OPT_GRAPH_TILES, 1)
    hb = engine.build_host_batch(b)
    x = rng.standard_normal((b.num_nodes, b.num_tags), dtype=np.float32) if opts.get("dense") else None
    db = eng.to_device(hb, x)
    rp, ci = hb.row_ptr.numpy(), hb.col_idx.numpy()
    val = None
    if opts.get("val") == "row":
        val = np.repeat((1.0 / np.maximum(np.diff(rp), 1)).astype(np.float32), np.diff(rp))
    elif opts.get("val") == "mixed":
        val = (rng.random(len(ci), dtype=np.float32) - 0.3).astype(np.float32)
    if val is not None:
        db.val = torch.from_numpy(val).cuda()
    embed = not opts.get("auto")
    n0 = eng.ctx.launches
    logits, probs, pred, emb = eng.forward(db, want_embed=embed)
    eng.ctx.synchronize()
    if opts.get("auto"):
        assert eng.ctx.launches - n0 == 1 + (x is not None)   # the whole classifier in one launch, behind a dense projection
    want_h, want = f64(b, rp, ci, val, x, opts.get("average", False))
    if embed:
        assert_close(emb.cpu().numpy(), want_h, "embeddings", scale=max(1.0, float(np.abs(want_h).max())))
    assert_close(logits.cpu().numpy(), want, "logits", scale=max(1.0, float(np.abs(want).max())))
    e = np.exp(want - want.max(1, keepdims=True))
    assert_close(probs.cpu().numpy(), e / e.sum(1, keepdims=True), "probs", scale=max(1.0, float(np.abs(want).max())))
    assert np.array_equal(pred.cpu().numpy(), logits.cpu().numpy().argmax(1))


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("sizes,degree", [([128], 6.0), ([0, 1, 0, 5, 1, 1, 0, 40, 128, 0, 3, 127, 1, 2], 2.2), ([1] * 300 + [2] * 10, 1.0),
                                          ([100, 7, 64, 30], 99.0), ([3, 1, 6, 2] * 2000, 2.0)], ids=lambda v: None)
def test_default_form(d, sizes, degree):
    """The form that small batches take by default: everything in one launch, with and without the node embeddings."""
    b = make(sizes, degree, d, 9, 4, 32 if d == 32 else 64, 2, seed=d + len(sizes))   # (hidden units whose sums fit the kernel's scratch)
    eng = engine.S2VInference(b.weights, b.levels)
    hb = engine.build_host_batch(b)
    db = eng.to_device(hb)
    n0 = eng.ctx.launches
    logits, _, _, emb = eng.forward(db, want_embed=True)
    again, _, _, _ = eng.forward(db)
    eng.ctx.synchronize()
    assert eng.ctx.launches - n0 == 2
    want_h, want = f64(b, hb.row_ptr.numpy(), hb.col_idx.numpy(), None, None, False)
    assert_close(emb.cpu().numpy(), want_h, "embeddings", scale=max(1.0, float(np.abs(want_h).max())))
    assert_close(logits.cpu().numpy(), want, "logits", scale=max(1.0, float(np.abs(want).max())))
    assert torch.equal(again, logits)


@pytest.mark.parametrize("auto", [False, True])                     # first level through the product table, and through the MMAs
@pytest.mark.parametrize("val", [None, "row", "mixed"])
@pytest.mark.parametrize("d,sizes,degree", [
    (64, [640, 100, 300, 0, 1], 30.0),                               # columns straight from global memory: more of them than a row has
    (32, [1024, 641, 3], 60.0),                                      # lanes (8, 16, 32), rows of 0, 1 and a few entries among them
    (128, [128, 1, 100, 7, 127], 60.0),
    (128, [33, 65, 2] * 40, 2.2), (64, [33, 65, 2] * 40, 2.2), (32, [33, 65, 2] * 40, 2.2),   # weights listed beside the columns
    (64, [90] * 400, 12.0),                                          # several tiles per CTA, lists used again
], ids=lambda v: None)
def test_fused_columns_and_weights_outside_and_inside_the_list(d, sizes, degree, val, auto):
    b = make(sizes, degree, d, 9, 3, 64, 3, seed=d + len(sizes))
    hb = engine.build_host_batch(b)
    eng = engine.S2VInference(b.weights, b.levels)
    if not auto:
        eng.ctx.set_option(eng.ctx.OPT_GRAPH_TILES, 1)
    db = eng.to_device(hb)
    rp, ci = hb.row_ptr.numpy(), hb.col_idx.numpy()
    v = None
    if val == "row":
        v = np.repeat((1.0 / np.maximum(np.diff(rp), 1)).astype(np.float32), np.diff(rp))
    elif val == "mixed":
        v = (np.random.default_rng(3).random(len(ci), dtype=np.float32) - 0.3).astype(np.float32)
    if v is not None:
        db.val = torch.from_numpy(v).cuda()
    logits, _, _, emb = eng.forward(db, want_embed=True)
    eng.ctx.synchronize()
    want_h, want = f64(b, rp, ci, v, None, False)
    assert_close(emb.cpu().numpy(), want_h, "embeddings", scale=max(1.0, float(np.abs(want_h).max())))
    assert_close(logits.cpu().numpy(), want, "logits", scale=max(1.0, float(np.abs(want).max())))


@pytest.mark.parametrize("d,hidden", [(32, 16), (32, 64), (64, 16), (64, 64), (128, 16)])
@pytest.mark.parametrize("graphs", [1, 9])
def test_pooled_sum_that_overflows(d, hidden, graphs):
    """One feature of one graph sums to infinity: the logits of the readout inside the kernel are those of the readout launch."""
    b = make([2] * graphs, 0, d, 3, 2, hidden, 3, seed=d)
    rng = np.random.default_rng(0)
    w_in = np.abs(b.weights["w_n2l"])
    w_in[1, 5] = 3e38
    w2 = np.abs(b.weights["h2_weight"])
    w2[:, 1] *= -1
    b.weights = dict(b.weights, w_n2l=w_in, h1_weight=np.abs(b.weights["h1_weight"]), h2_weight=w2)
    b.tags = rng.integers(0, 1, 2 * graphs).astype(np.int32)
    b.tags[:2] = 1
    got = {}
    for mode in (0, 2):
        eng = engine.S2VInference(b.weights, b.levels)
        eng.ctx.set_option(eng.ctx.OPT_GRAPH_TILES, mode)
        logits, _, pred, _ = eng.forward(eng.to_device(engine.build_host_batch(b)))
        eng.ctx.synchronize()
        got[mode] = logits.cpu().numpy(), pred.cpu().numpy()
    assert np.array_equal(np.isposinf(got[0][0][0]), [True, False, True]) and np.isneginf(got[0][0][0, 1])
    np.testing.assert_allclose(got[2][0], got[0][0], rtol=1e-5, atol=1e-5)
    assert np.array_equal(got[2][1], got[0][1])


def test_fused_reports_a_graph_beyond_the_hint_and_an_edge_between_graphs():
    b = make([30, 300, 25], 2.0, 64, 5, 2, 64, 2, seed=1)
    eng = engine.S2VInference(b.weights, b.levels)
    db = eng.to_device(engine.build_host_batch(b))
    db.max_graph_nodes = 100                            # understated: tiles of 128 rows
    eng.forward(db)
    with pytest.raises(capi.S2VError) as e:
        eng.ctx.synchronize()
    assert e.value.status in (-2, -4)
    db.max_graph_nodes = 300
    eng.forward(db)
    eng.ctx.synchronize()                               # the context carries on
    ci = db.col_idx.clone()
    ci[0] = b.num_nodes - 1
    db.col_idx = ci
    eng.forward(db)
    with pytest.raises(capi.S2VError) as e:
        eng.ctx.synchronize()
    assert e.value.status == -4


@pytest.mark.parametrize("graphs", [189, 190])   # d = 32, 600 nodes each: the last batch of one round of tiles, and one beyond it
def test_large_d32_batches(graphs):
    b = make([600] * graphs, 6.5, 32, 5, 3, 64, 2, seed=graphs)
    eng = engine.S2VInference(b.weights, b.levels)
    hb = engine.build_host_batch(b)
    db = eng.to_device(hb)
    n0 = eng.ctx.launches
    logits, _, _, _ = eng.forward(db)
    eng.ctx.synchronize()
    assert eng.ctx.launches - n0 == (4 if graphs == 189 else 6)
    _, want = f64(b, hb.row_ptr.numpy(), hb.col_idx.numpy(), None, None, False)
    assert_close(logits.cpu().numpy(), want, "logits", scale=max(1.0, float(np.abs(want).max())))
