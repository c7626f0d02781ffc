"""GPU: rows that hold the lowest finite values, -inf or NaN, against the same operation in float64.

A masked position is either -inf or the type's lowest finite value; both must act as "contributes nothing" wherever any
other value is larger, and a NaN must not vanish.
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def masked_logits(V, dtype, dev):
    """One row per kind of masking, [rows, V]; the target of every row is column 1."""
    x = torch.randn(8, V, device=dev, generator=torch.Generator(device=dev).manual_seed(V)).mul_(2).to(dtype)
    low = torch.finfo(dtype).min
    x[0, V // 2:] = low            # whole shares and whole vectors of the lowest value, behind and before the kept ones
    x[1, 2:V // 2] = low
    x[2, V // 2:] = -math.inf
    x[3, 3 * V // 4:] = math.nan   # a share that holds nothing but NaN
    x[4, 2:V // 2] = -math.inf
    x[4, V // 4] = math.nan        # one NaN among masked logits
    x[5] = low                     # nothing but the lowest value: uniform
    x[6] = 3e38                    # so large that x * log2(e) overflows: uniform
    x[7, 2:] = -math.inf           # two logits are left
    return x


# block kernel: short rows and rows of more than 800 KB; cluster kernel: 1, 2, 4 and 8 CTAs per row, rows of whole and of
# partial vectors; in place (the training step's form) always the block kernel
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [50, 5000, 5001, 9000, 32000, 50257, 151936, 420001])
@pytest.mark.parametrize("in_place", [False, True])
def test_cross_entropy_of_masked_logits(cuda_device, dtype, V, in_place):
    from metal_candle_b200 import _lib, backend
    from metal_candle_b200.training import cross_entropy_loss

    x = masked_logits(V, dtype, cuda_device)
    lib = _lib.load()
    for row in range(x.shape[0]):
        r64 = x[row].double()
        # log_softmax by hand: the largest logit first, so that nothing overflows
        d = r64 - r64[~r64.isnan()].max()
        logp = d - d.exp().sum().log()
        want, want_g = -logp[1], logp.exp()
        want_g[1] -= 1.0
        if in_place:
            g = x[row].clone()
            t = torch.ones(1, dtype=torch.int32, device=cuda_device)
            nll, count, loss = torch.empty(1, device=cuda_device), torch.empty_like(t), torch.empty(2, device=cuda_device)
            _lib.check(lib.mcb_cross_entropy(g.data_ptr(), t.data_ptr(), nll.data_ptr(), count.data_ptr(), loss.data_ptr(), 1, V, 1,
                                             backend._dtype_code(g), backend._stream()))
        else:
            t = torch.ones(1, 1, dtype=torch.int64, device=cuda_device)
            loss, g = cross_entropy_loss(x[row].clone().view(1, 1, V), t, return_grad=True)
            g = g.view(-1)
        if want.isnan():
            assert loss[0].isnan() and g.isnan().all(), row
            continue
        # float32 sums of exponentials of 2^-22 each; a gradient element is rounded to its type once
        assert abs(float(loss[0]) - float(want)) <= 1e-5 * abs(float(want)) + 1e-6, (row, float(loss[0]), float(want))
        rel = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-5
        assert ((g.double() - want_g).abs() <= rel * want_g.abs() + 1e-7).all(), row
    assert _lib.device_status() == 0


# rows of whole and of partial 16-byte vectors, held in registers and streamed
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("seq", [64, 65, 776, 777, 1030, 2100])
@pytest.mark.parametrize("scale", [0.125, 0.0, -0.5])
def test_causal_softmax_of_any_scale(cuda_device, dtype, seq, scale):
    from metal_candle_b200 import _lib, backend

    rows = 2 * seq
    x = torch.randn(rows, seq, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(seq)).mul_(4).to(dtype)
    y = torch.full_like(x, math.nan)
    _lib.check(_lib.load().mcb_softmax_causal_fwd(x.data_ptr(), y.data_ptr(), rows, seq, seq, scale, backend._dtype_code(x), backend._stream()))
    mask = torch.ones(seq, seq, dtype=torch.bool, device=cuda_device).triu(1).repeat(2, 1)
    want = torch.softmax((x.double() * scale).masked_fill(mask, -math.inf), -1)
    # bfloat16: rounded to its type once; float32: exponents up to 40, each product and difference rounded to 2^-24 of that
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    assert ((y.double() - want).abs() <= rel * want + 1e-30).all()


# rows held in registers (1 to 8 vectors per lane), streamed rows, register kernels; whole and partial vectors
SOFTMAX_WIDTHS = [64, 65, 300, 776, 777, 1040, 1041, 2050, 2104, 4097]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", SOFTMAX_WIDTHS)
@pytest.mark.parametrize("causal", [False, True])
def test_softmax_of_the_largest_values(cuda_device, dtype, D, causal):
    """Scores whose product with log2(e) overflows: rows masked with the lowest value, wholly and in part."""
    from metal_candle_b200 import _lib, backend

    low, rows = torch.finfo(dtype).min, D if causal else 96
    x = torch.randn(rows, D, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(D)).to(dtype)
    kinds = [low, 3e38, -2.5e38]
    for i, value in enumerate(kinds):
        x[i::8] = value
    x[3::8, :D // 2] = low
    x[4::8, 1:] = low
    x[5::8, D // 3] = 3e38
    y = torch.full_like(x, math.nan)
    x64 = x.double()
    if causal:
        _lib.check(_lib.load().mcb_softmax_causal_fwd(x.data_ptr(), y.data_ptr(), rows, D, D, 1.0, backend._dtype_code(x), backend._stream()))
        x64 = x64.masked_fill(torch.ones(D, D, dtype=torch.bool, device=cuda_device).triu(1), -math.inf)
    else:
        backend.softmax_fused(x, out=y)
    want = torch.softmax(x64, -1)
    rel = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    assert ((y.double() - want).abs() <= rel * want + 1e-30).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", SOFTMAX_WIDTHS)
def test_softmax_keeps_nan_and_clears_masked_rows(cuda_device, dtype, D):
    from metal_candle_b200 import backend

    x = torch.randn(96, D, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(D)).to(dtype)
    x[0::4] = math.nan
    x[1::4] = -math.inf
    x[2::4] = -math.inf
    x[2::4, D // 2] = math.nan
    y = backend.softmax_fused(x)
    assert y[0::4].isnan().all()
    assert (y[1::4] == 0).all()                     # nothing kept: zeros
    assert y[2::4, D // 2].isnan().all()
    torch.testing.assert_close(y[3::4].double(), torch.softmax(x[3::4].double(), -1), rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-5, atol=1e-30)
