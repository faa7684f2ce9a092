"""Weights and embeddings of uneven size through the kernel that keeps whole graphs in shared memory (graph_fused.cu), against a
float64 restatement of the classifier (kernel_mean_field.cpp:28-47), judged feature by feature: a feature a millionth or a billionth
the size of its neighbours has to keep its digits."""
import numpy as np
import pytest

from graphnn_b200 import engine
from test_graph_fused_gpu import f64, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["small", "large"])          # W converted by every CTA, or once in front
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("span", [0, 12, 24, 40])
@pytest.mark.parametrize("kind", ["columns", "units"])
def test_features_of_uneven_size(kind, span, d, form):
    b = make([20, 128, 1, 33, 90] * 3, 2.2, d, 9, 3, 64, 2, seed=d + span)
    rng = np.random.default_rng(span)
    c = np.exp2(-rng.integers(0, span + 1, d)).astype(np.float32)
    c[:2] = 1.0, 2.0 ** -span
    w = b.weights["p_node_conv"] * c                           # output features of size c ...
    if kind == "units":                                        # ... and weights that undo it, so that all of them count in every sum
        w = w / c[:, None]
    b.weights = dict(b.weights, p_node_conv=w.astype(np.float32), w_n2l=(b.weights["w_n2l"] * c).astype(np.float32))
    hb = engine.build_host_batch(b)
    eng = engine.S2VInference(b.weights, b.levels)
    eng.ctx.set_option(eng.ctx.OPT_GRAPH_TILES, 1 if form == "large" else 2)
    _, _, _, emb = eng.forward(eng.to_device(hb), want_embed=True)
    eng.ctx.synchronize()
    want, _ = f64(b, hb.row_ptr.numpy(), hb.col_idx.numpy(), None, None, False)
    size = np.abs(want).max(0)
    assert (size > 0).sum() > d // 2
    err = np.abs(emb.cpu().numpy() - want).max(0)[size > 0] / size[size > 0]
    # sums of d products in 22 bits, three levels of them: about 3e-7; 1e-5 is the bar of the path
    assert err.max() < 2e-6, f"feature error up to {err.max():.1e}"


@pytest.mark.parametrize("d", [32, 64, 128])
def test_infinite_weight_spoils_its_feature_only(d):
    b = make([20, 40, 7], 2.2, d, 9, 1, 64, 2, seed=d)
    w = b.weights["p_node_conv"].copy()
    w[3, 5] = np.inf
    b.weights = dict(b.weights, p_node_conv=w)
    hb = engine.build_host_batch(b)
    eng = engine.S2VInference(b.weights, b.levels)
    eng.ctx.set_option(eng.ctx.OPT_GRAPH_TILES, 1)
    eng.ctx.set_option(eng.ctx.OPT_FIRST_LEVEL_TABLE, 0)       # the level through the products
    _, _, _, emb = eng.forward(eng.to_device(hb), want_embed=True)
    eng.ctx.synchronize()
    b.weights = dict(b.weights, p_node_conv=np.where(np.isinf(w), 0, w))
    want, _ = f64(b, hb.row_ptr.numpy(), hb.col_idx.numpy(), None, None, False)
    emb = emb.cpu().numpy()
    keep = np.arange(d) != 5
    assert np.abs(emb[:, keep] - want[:, keep]).max() < 1e-5 * max(1.0, np.abs(want).max())
    assert not np.isfinite(emb[:, 5]).all()
