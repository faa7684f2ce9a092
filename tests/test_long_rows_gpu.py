"""GPU parity of the level kernels on rows that are summed ahead of the main loop (long_rows.cuh): lengths around the
limits, several in one group of rows, with and without weights, on both level kernels, against float64."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from conftest import assert_close
from graphnn_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tc", [0, 2])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("rp64", [False, True])
@pytest.mark.parametrize("weights,x", [(False, True), (True, False)])
def test_long_rows(tc, d, rp64, weights, x):
    rng = np.random.default_rng(d)
    n, n_src = 2500, 4000
    deg = rng.integers(0, 9, n)
    for i, k in enumerate([255, 256, 257, 300, 2047, 2048, 2049, 5000, 9001]):
        deg[[3, 5, 6, 130, 131, 255, 256, 1700, n - 1][i]] = k
    row_ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64 if rp64 else np.int32)
    nnz = int(row_ptr[-1])
    col = rng.integers(0, n_src, nnz).astype(np.int32)
    val = rng.standard_normal(nnz).astype(np.float32) if weights else None
    H = rng.standard_normal((n_src, d), dtype=np.float32)
    W = rng.standard_normal((d, d), dtype=np.float32) * 0.1
    X = rng.standard_normal((n, d), dtype=np.float32) if x else None
    S = np.zeros((n, d))
    np.add.at(S, np.repeat(np.arange(n), deg), H[col].astype(np.float64) * (1.0 if val is None else val[:, None].astype(np.float64)))
    want = np.maximum(S @ W.astype(np.float64) + (0 if X is None else X), 0)
    ctx = capi.Context(0)
    ctx.set_option(ctx.OPT_LEVEL_TC, tc)
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()
    out = torch.full((n, d), float("nan"), device="cuda")
    args = [dev(a) for a in (row_ptr, col, val, H, W, X)]
    torch.cuda.synchronize()
    mag = np.maximum(np.abs(want).max(1, keepdims=True), 1)   # hub sums are held to 1e-5 of their row's scale
    for _ in range(2):                                        # twice: the second time `out` holds results
        ctx.level(*args, out)
        ctx.synchronize()
        assert_close(out.cpu().numpy() / mag, want / mag, "level")
    if X is not None:                                         # X in place: the row's term and its result share memory
        ctx.level(*args[:5], args[5], args[5])
        ctx.synchronize()
        assert_close(args[5].cpu().numpy() / mag, want / mag, "level, X in place")


@pytest.mark.parametrize("tc,d,rp64,weights,x", [(2, 64, False, False, True), (2, 64, False, True, False), (2, 128, False, True, True),
                                                 (2, 128, False, False, False), (0, 32, False, True, True), (0, 32, True, False, False),
                                                 (0, 64, True, True, True), (0, 128, True, False, True)])
@pytest.mark.parametrize("hubs", [False, True])
def test_long_rows_in_front(tc, d, rp64, weights, x, hubs):
    """Levels large enough for the sums to be a kernel of their own: rows at both ends, several in a group, the level before and the
    level behind on the same stream (each reads what the other wrote)."""
    rng = np.random.default_rng(d + hubs)
    n = 160000 + 77
    deg = rng.integers(0, 3, n)
    if hubs:
        for r, k in [(0, 300), (1, 2049), (6, 257), (130, 5000), (131, 256), (80000, 9001), (n - 2, 700), (n - 1, 2500)]:
            deg[r] = k
    row_ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64 if rp64 else np.int32)
    nnz = int(row_ptr[-1])
    col = rng.integers(0, n, nnz).astype(np.int32)
    col[row_ptr[5]:row_ptr[6]] = 0                             # rows that read what a hub row became a level earlier
    val = rng.standard_normal(nnz).astype(np.float32) if weights else None
    H = rng.standard_normal((n, d), dtype=np.float32)
    W = rng.standard_normal((d, d), dtype=np.float32) * 0.02
    X = rng.standard_normal((n, d), dtype=np.float32) if x else None
    A = sp.csr_matrix((np.ones(nnz) if val is None else val.astype(np.float64), col, row_ptr), shape=(n, n))
    ctx = capi.Context(0)
    ctx.set_option(ctx.OPT_LEVEL_TC, tc)
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()
    h0, rp, ci, vl, w, xx = (dev(a) for a in (H, row_ptr, col, val, W, X))
    h1, h2 = torch.full((n, d), float("nan"), device="cuda"), torch.full((n, d), float("nan"), device="cuda")
    torch.cuda.synchronize()
    for _ in range(2):
        ctx.level(rp, ci, vl, h0, w, xx, h1)
        ctx.level(rp, ci, vl, h1, w, xx, h2)
    ctx.synchronize()
    for src, got in ((H, h1), (h1.cpu().numpy(), h2)):
        want = np.maximum((A @ src.astype(np.float64)) @ W.astype(np.float64) + (0 if X is None else X), 0)
        mag = np.maximum(np.abs(want).max(1, keepdims=True), 1)
        assert_close(got.cpu().numpy() / mag, want / mag, "level")
