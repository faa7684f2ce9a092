"""Large matrices with few entries a row at d = 128 (level_tc.cu): the forward of a batch that may hold hubs and of one that cannot, against float64."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from graphnn_b200 import engine

pytestmark = pytest.mark.gpu
LEAST = 131072


def sparse_rows(n, seed, hubs):
    rng = np.random.default_rng(seed)
    deg = rng.integers(0, 4, n)
    if hubs:
        lengths = [127, 128, 129, 255, 256, 257, 300, 1023, 2047, 2048, 2049, 5000]
        deg[rng.permutation(np.arange(100, n - 100))[:12]] = lengths
        deg[[0, 1, 9, n - 1]] = [700, 300, 258, 3000]
        deg[60000:60040] = 270
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    return deg, rp, rng.integers(0, n, int(rp[-1])).astype(np.int32), rng


@pytest.mark.parametrize("x", [False, True])
@pytest.mark.parametrize("weights", [False, True])
def test_level(gpu_ctx, x, weights):
    """One level with the count known (level_tc.cu), and as the entry without it takes it (level_stream.cu)."""
    d, n = 128, LEAST + 50
    deg, rp, col, rng = sparse_rows(n, 11, True)
    val = rng.standard_normal(col.size).astype(np.float32) if weights else None
    H, W = rng.standard_normal((n, d), dtype=np.float32), rng.standard_normal((d, d), dtype=np.float32) * 0.1
    X = rng.standard_normal((n, d), dtype=np.float32) if x else None
    A = sp.csr_matrix((np.ones(col.size) if val is None else val.astype(np.float64), col, rp), (n, n))
    want = np.maximum(A @ H.astype(np.float64) @ W.astype(np.float64) + (0 if X is None else X), 0)
    rows = np.maximum(np.abs(want).max(1, keepdims=True), 1)   # hub sums are held to 1e-5 of their row's scale
    args = [None if a is None else torch.from_numpy(a).cuda() for a in (rp, col, val, H, W, X)]
    ptr = lambda t: None if t is None else t.data_ptr()
    for known in (True, False):
        out = torch.full((n, d), float("nan"), device="cuda")
        torch.cuda.synchronize()
        if known:
            gpu_ctx.level(*args, out)
        else:
            gpu_ctx.call("s2v_level_f32", None, n, n, d, *map(ptr, args), ptr(out))
        gpu_ctx.synchronize()
        np.testing.assert_allclose(out.cpu().numpy() / rows, want / rows, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("hubs", [False, True])
@pytest.mark.parametrize("weights", [False, True])
def test_forward(hubs, weights):
    d, n, tags, levels, graphs = 128, LEAST + 37, 9, 3, 97
    deg, rp, col, rng = sparse_rows(n, 3 + hubs, hubs)
    val = (0.2 + rng.random(col.size, dtype=np.float32)) if weights else None
    tag = rng.integers(0, tags, n).astype(np.int32)
    gp = np.sort(np.concatenate([[0, n], rng.integers(0, n, graphs - 1)])).astype(np.int32)
    w = {k: rng.standard_normal(s).astype(np.float32) * 0.05 for k, s in
         {"w_n2l": (tags, d), "p_node_conv": (d, d), "h1_weight": (d, 64), "h2_weight": (64, 2)}.items()}
    eng = engine.S2VInference(w, levels)
    eng.ctx.set_option(eng.ctx.OPT_GRAPH_TILES, 0)
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()
    launches = {}
    A = sp.csr_matrix((np.ones(col.size) if val is None else val.astype(np.float64), col, rp), (n, n))
    x = w["w_n2l"].astype(np.float64)[tag]
    h = np.maximum(x, 0)
    for _ in range(levels):
        h = np.maximum(A @ h @ w["p_node_conv"].astype(np.float64) + x, 0)
    rows = np.maximum(np.abs(h).max(1, keepdims=True), 1)   # what passes through a hub is held to 1e-5 of its row's scale
    for largest in (0, 2048):   # unknown; no graph, and so no row, of more
        db = engine.DeviceBatch(graphs, n, dev(rp), dev(col), dev(gp), dev(tag), None, dev(val), largest)
        n0 = eng.ctx.launches
        _, _, _, embed = eng.forward(db, want_embed=True)
        eng.ctx.synchronize()
        launches[largest] = eng.ctx.launches - n0
        np.testing.assert_allclose(embed.cpu().numpy() / rows, h / rows, rtol=1e-5, atol=1e-5)
    assert launches[0] - launches[2048] == levels - 1   # the kernel in front, where there may be hubs
