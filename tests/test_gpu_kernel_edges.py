"""GPU parity at the sizes where the kernels' tiles, splits and dispatch rules have their edges, against the CPU oracle.

Tolerances, max|gpu - oracle| / max|oracle|: 1e-4 for float32 and 2e-2 for bfloat16, the bounds of the other parity
tests (float32: a reduction of k terms of size s carries at most about k 2^-24 s, which is 1e-4 of the largest output
at the 1500 terms used here; bfloat16: operands and results rounded to 2^-9 relative).
"""
import numpy as np
import pytest
import torch

from oracle import reference_ops as R
from oracle import seeded as S

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 1e-4, torch.bfloat16: 2e-2}


def dev_t(a, dtype, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev).to(dtype).contiguous()


def back(t):
    return t.detach().float().cpu().numpy()


def rounded(a, dtype):
    return a if dtype == torch.float32 else S.bf16_round(a)


# float32: 128 x 64 tiles, reductions split in 2 to 8, rank columns through the lean kernels (below 24) and the tile
# kernel, odd strides
@pytest.mark.parametrize("M,K,N,r", [(1, 3, 5, 1), (127, 33, 65, 3), (129, 511, 63, 23), (512, 768, 768, 24), (1030, 129, 257, 40),
                                     (2000, 1500, 1, 1), (64, 1500, 300, 65)])
def test_f32_linear_edges(cuda_device, M, K, N, r):
    from metal_candle_b200 import backend as B

    r = min(r, K, N)
    c = S.lora_linear_case(31, M, K, N, r)
    x, W, dy, A, Bm = (dev_t(c[k], torch.float32, cuda_device) for k in ("x", "W", "dy", "A", "B"))
    y, h = B.lora_linear_forward(x, W, None, A, Bm, 2.0)
    want_y, want_h = R.lora_linear_forward(c["x"], c["W"], None, c["A"], c["B"], 2.0)
    assert R.max_abs_normalised(back(y), want_y) <= 1e-4
    assert R.max_abs_normalised(back(h)[:r, :M].T, 2.0 * want_h) <= 1e-4
    want = R.lora_linear_backward(c["x"], c["W"], c["A"], c["B"], 2.0, c["dy"])
    from metal_candle_b200._lib import MCB_W_OUT_IN
    for wt, kw in ((B.transpose_2d(W), {}), (W, dict(weight_layout=MCB_W_OUT_IN))):
        got = B.lora_linear_backward(x, wt, A, Bm, 2.0, dy, h_save=h, **kw)
        for g, w in zip(got, want):
            assert R.max_abs_normalised(back(g), w) <= 1e-4


# the cluster kernel of the delta: one and four tokens per cluster, its last token count (256 bf16, 512 float32) and the
# first one beyond, ranks with and without the shuffle reduction, more columns than CTAs and fewer
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,K,N,r", [(1, 512, 512, 8), (1, 8, 8, 1), (18, 1024, 72, 8), (19, 1024, 72, 8), (5, 4096, 264, 64), (3, 96, 48, 24),
                                     (256, 264, 520, 16), (257, 264, 520, 16), (512, 64, 64, 4), (513, 64, 64, 4)])
def test_delta_edges(cuda_device, dtype, M, K, N, r):
    from metal_candle_b200 import backend as B

    c = S.lora_linear_case(32, M, K, N, r)
    x = rounded(c["x"], dtype)
    got = B.lora_forward_fused(dev_t(x, dtype, cuda_device), dev_t(c["A"], torch.float32, cuda_device), dev_t(c["B"], torch.float32, cuda_device), 2.0)
    want, _ = R.lora_forward(x, rounded(c["A"], dtype), rounded(c["B"], dtype), 2.0)
    assert R.max_abs_normalised(back(got), want) <= TOL[dtype]
