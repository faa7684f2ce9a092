"""Dense input projection: the tiled kernel (d = 32, 64, 128) at row counts around its tiles, against the plain one's order of
sums restated in float64."""
import numpy as np
import pytest
import torch

from conftest import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,F", [(32, 1), (32, 21), (64, 3), (64, 37), (128, 82), (128, 5), (48, 7)])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 129, 5000])
def test_input_proj_dense(gpu_ctx, d, F, n):
    rng = np.random.default_rng(n + d)
    X, W = rng.standard_normal((n, F), dtype=np.float32), rng.standard_normal((F, d), dtype=np.float32)
    msg, h0 = torch.full((n, d), float("nan"), device="cuda"), torch.full((n, d), float("nan"), device="cuda")
    gpu_ctx.input_proj_dense(torch.from_numpy(X).cuda(), torch.from_numpy(W).cuda(), msg, h0)
    gpu_ctx.synchronize()
    want = X.astype(np.float64) @ W.astype(np.float64)
    assert_close(msg.cpu().numpy(), want, "msg", scale=10)
    assert torch.equal(h0, torch.clamp(msg, min=0))
