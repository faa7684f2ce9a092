"""Large levels (level_stream.cu): row lengths around the limits between the gather, a warp and a whole CTA per row, ragged last tiles, weights,
the forms of X, 64-bit offsets, fewer SMs, infinities, against float64."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from graphnn_b200 import capi

pytestmark = pytest.mark.gpu
LEAST = 131072   # rows from which the kernel is taken


def problem(d, n, seed, hubs=True):
    rng = np.random.default_rng(seed)
    n_src = 5000
    deg = rng.integers(0, 9, n)
    deg[:64] = 0                                                  # whole units without an entry
    if hubs:
        at = rng.permutation(np.arange(64, n - 3))[:20]
        deg[at] = [127, 128, 129, 130, 255, 256, 257, 300, 1023, 1024, 1025, 2047, 2048, 2049, 2050, 5000, 16, 17, 33, 65]
        deg[[n - 1, n - 2, 64, 65]] = [3000, 129, 128, 129]
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    col = rng.integers(0, n_src, int(rp[-1])).astype(np.int32)
    val = rng.standard_normal(col.size).astype(np.float32)
    H = rng.standard_normal((n_src, d), dtype=np.float32)
    W = rng.standard_normal((d, d), dtype=np.float32) * 0.1
    return deg, rp, col, val, H, W, rng


def reference(deg, rp, col, val, H, W, X):
    """The level in float64, and what fp32 may be off by: deg additions and d products and additions at 2^-24 each, and 2^-21 for the three
    TF32 products, all relative to the sums of magnitudes."""
    v = np.ones(col.size) if val is None else val.astype(np.float64)
    H, W = H.astype(np.float64), W.astype(np.float64)
    x = 0.0 if X is None else X.astype(np.float64)
    shape = (rp.size - 1, H.shape[0])
    want = sp.csr_matrix((v, col, rp), shape) @ H @ W + x
    mag = sp.csr_matrix((np.abs(v), col, rp), shape) @ np.abs(H) @ np.abs(W)
    bound = mag * ((deg[:, None] + H.shape[1]) * 2.0 ** -24 + 2.0 ** -21) + (np.abs(want) + np.abs(x)) * 2.0 ** -23
    return np.where(want < 0, 0, want), bound


def check(out, want, bound):
    err = np.abs(out.cpu().numpy().astype(np.float64) - want)
    assert (err <= bound).all(), f"{(err > bound).sum()} elements off, worst {np.nanmax(err / bound)} of the bound"


dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("n", [LEAST, LEAST + 1, LEAST + 77])
@pytest.mark.parametrize("weights,x,rp64", [(False, True, False), (True, False, True), (True, True, False)])
def test_level(gpu_ctx, d, n, weights, x, rp64):
    deg, rp, col, val, H, W, rng = problem(d, n, d + n)
    val = val if weights else None
    X = rng.standard_normal((n, d), dtype=np.float32) if x else None
    want, bound = reference(deg, rp, col, val, H, W, X)
    args = [dev(a) for a in (rp.astype(np.int64) if rp64 else rp, col, val, H, W, X)]
    out = torch.full((n, d), float("nan"), device="cuda")
    gpu_ctx.level(*args, out)
    gpu_ctx.synchronize()
    check(out, want, bound)
    if x:   # X in place
        gpu_ctx.level(*args, args[5])
        gpu_ctx.synchronize()
        assert torch.equal(args[5], out)


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("weights", [False, True])
@pytest.mark.parametrize("together", [7, 8, 40])
def test_long_rows_of_one_block(gpu_ctx, d, weights, together):
    """Long rows next to each other: few (the whole CTA on each) and many (a warp on each), lengths around the stages of the ring."""
    n = LEAST + 5
    deg, rp, col, val, H, W, rng = problem(d, n, d + together, hubs=False)
    lengths = [256, 257, 319, 320, 321, 512, 1023, 1025, 129, 16 * 32 * 32 + 1, 2048, 2049, 640, 1984, 2047]
    deg[70000:70000 + together] = [lengths[i % len(lengths)] for i in range(together)]
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    col = rng.integers(0, H.shape[0], int(rp[-1])).astype(np.int32)
    val = rng.standard_normal(col.size).astype(np.float32) if weights else None
    want, bound = reference(deg, rp, col, val, H, W, None)
    out = torch.full((n, d), float("nan"), device="cuda")
    gpu_ctx.level(dev(rp), dev(col), dev(val), dev(H), dev(W), None, out)
    gpu_ctx.synchronize()
    check(out, want, bound)


def test_one_long_row_is_as_fast_per_byte_at_d_128(gpu_ctx):
    """(1.84 times the time of d = 64 with stages of 32 rows and 96 rows on their way; 1.41 now, through the kernel in front of level_tc.cu, which
    a matrix with so few entries a row takes at d = 128, 1.34 through level_stream.cu; H does not fit the L2)"""
    n, long = 4 * LEAST, 2 * LEAST
    gen = torch.Generator(device="cuda").manual_seed(1)
    deg = torch.ones(n, dtype=torch.int64, device="cuda")
    deg[77] = long
    rp = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    rp[1:] = deg.cumsum(0)
    col = torch.randint(0, n, (int(rp[-1]),), generator=gen, device="cuda", dtype=torch.int32)
    least = {}
    for d in (64, 128):
        H, W, out = torch.randn((n, d), device="cuda"), torch.randn((d, d), device="cuda"), torch.empty((n, d), device="cuda")
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(s)
            gpu_ctx.level(rp, col, None, H, W, None, out, stream=s.cuda_stream)
            b.record(s)
            b.synchronize()
            times.append(a.elapsed_time(b))
        least[d] = min(times)
    assert least[128] < 1.6 * least[64], least


@pytest.mark.parametrize("d", [32, 64, 128])
def test_forms(gpu_ctx, d):
    """The same rows through a graph (twice), with SMs left to others, and with X from a table: the same bits."""
    n, tags = LEAST + 19, 5
    deg, rp, col, val, H, W, rng = problem(d, n, d)
    table, idx = rng.standard_normal((tags, d), dtype=np.float32), rng.integers(0, tags, n).astype(np.int32)
    want, bound = reference(deg, rp, col, None, H, W, table[idx])
    rp, col, H, W, table, idx = [dev(a) for a in (rp, col, H, W, table, idx)]
    X = table[idx.long()].contiguous()
    out = [torch.full((n, d), float("nan"), device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    gpu_ctx.level(rp, col, None, H, W, X, out[0])
    gpu_ctx.level_lookup(rp, col, None, H, W, table, idx, out[1])
    gpu_ctx.synchronize()
    gpu_ctx.set_option(gpu_ctx.OPT_RESERVED_SMS, 20)
    try:
        gpu_ctx.level(rp, col, None, H, W, X, out[2])
        gpu_ctx.synchronize()
    finally:
        gpu_ctx.set_option(gpu_ctx.OPT_RESERVED_SMS, 0)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        gpu_ctx.level(rp, col, None, H, W, X, out[3], stream=s.cuda_stream)
        out[3].mul_(1.0)   # behind the level: counts on the rows of the kernel in front too
    for _ in range(2):
        out[3].fill_(float("nan"))
        g.replay()
    torch.cuda.synchronize()
    check(out[0], want, bound)
    for o in out[1:]:
        assert torch.equal(o, out[0])


@pytest.mark.parametrize("d", [32, 64, 128])
def test_infinities_stay_in_their_rows(gpu_ctx, d):
    n = LEAST + 3
    deg, rp, col, val, H, W, rng = problem(d, n, 7, hubs=False)
    H[0] = np.inf            # (row 0 is also what lanes past the end of a row read)
    H[1] = np.nan
    touched = sp.csr_matrix((np.isin(col, [0, 1]).astype(np.int32), col, rp), (n, H.shape[0])).sum(1).A1 > 0
    clean = H.copy()
    clean[:2] = 0
    want, bound = reference(deg, rp, col, None, clean, W, None)
    out = torch.zeros((n, d), device="cuda")
    gpu_ctx.level(dev(rp), dev(col), None, dev(H), dev(W), None, out)
    gpu_ctx.synchronize()
    out = out.cpu().numpy()
    assert touched.any() and not np.isfinite(out[touched]).all(1).any()
    assert (np.abs(out[~touched] - want[~touched]) <= bound[~touched]).all()


def test_no_entries(gpu_ctx):
    n, d = LEAST, 64
    X = torch.randn((n, d), device="cuda")
    out = torch.full((n, d), float("nan"), device="cuda")
    gpu_ctx.level(torch.zeros(n + 1, dtype=torch.int32, device="cuda"), torch.zeros(0, dtype=torch.int32, device="cuda"), None,
                  torch.zeros((0, d), device="cuda"), torch.randn((d, d), device="cuda"), X, out)
    gpu_ctx.synchronize()
    assert torch.equal(out, torch.where(X < 0, torch.zeros_like(X), X))
