"""Large levels with SMs left to others (level_stream.cu, one CTA per SM): the same bits as on the whole GPU, and no slower than the SMs that are
left explain."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LEAST = 131072


@pytest.fixture
def reserve(gpu_ctx):
    yield lambda n: gpu_ctx.set_option(gpu_ctx.OPT_RESERVED_SMS, n)
    gpu_ctx.set_option(gpu_ctx.OPT_RESERVED_SMS, 0)


def matrix(n, gen, hubs, mean=8):
    deg = torch.randint(0, 2 * mean + 1, (n,), generator=gen, device="cuda")
    deg[:64] = 0
    if hubs:
        lengths = torch.tensor([7, 8, 9, 15, 16, 17, 31, 33, 63, 65, 127, 128, 129, 257, 1025, 2049, 5000], device="cuda")
        deg[100:100 + lengths.numel()] = lengths
        deg[-1] = 129
    rp = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    rp[1:] = deg.cumsum(0)
    return rp, torch.randint(0, n, (int(rp[-1]),), generator=gen, device="cuda", dtype=torch.int32)


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("weights,x,rp64,table", [(False, True, False, False), (True, False, True, False), (True, True, False, False), (False, False, False, True)])
def test_same_bits(gpu_ctx, reserve, d, weights, x, rp64, table):
    n, gen = LEAST + 13, torch.Generator(device="cuda").manual_seed(d)
    rp, col = matrix(n, gen, True)
    rand = lambda *s: torch.randn(s, generator=gen, device="cuda")
    val, H, W, X = rand(col.numel()) if weights else None, rand(n, d), rand(d, d), rand(n, d) if x else None
    tab, idx = rand(5, d), torch.randint(0, 5, (n,), generator=gen, device="cuda", dtype=torch.int32)
    rp = rp.long() if rp64 else rp
    torch.cuda.synchronize()
    outs = []
    for left in (0, 1, 20, torch.cuda.get_device_properties(0).multi_processor_count - 1):
        reserve(left)
        out = torch.full((n, d), float("nan"), device="cuda")
        torch.cuda.synchronize()
        if table:
            gpu_ctx.level_lookup(rp, col, val, H, W, tab, idx, out)
        else:
            gpu_ctx.level(rp, col, val, H, W, X, out)
        gpu_ctx.synchronize()
        outs.append(out)
    assert torch.isfinite(outs[0]).all()
    for out in outs[1:]:
        assert torch.equal(out, outs[0])


@pytest.mark.parametrize("d", [32, 64])
def test_one_reserved_sm_does_not_cost_half_the_gather(gpu_ctx, reserve, d):
    """(1.70 times the time of the whole GPU with one of the two CTAs per SM, 1.09 now)"""
    n, gen = 1 << 20, torch.Generator(device="cuda").manual_seed(3)
    rp, col = matrix(n, gen, False)
    H, W, out = torch.randn((n, d), device="cuda"), torch.randn((d, d), device="cuda"), torch.empty((n, d), device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    least = []
    for left in (0, 1):
        reserve(left)
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(s)
            gpu_ctx.level(rp, col, None, H, W, None, out, stream=s.cuda_stream)
            b.record(s)
            b.synchronize()
            times.append(a.elapsed_time(b))
        least.append(min(times))
    assert least[1] < 1.35 * least[0], least
