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


# float32: 128 x 128 and 128 x 64 tiles, reductions split in up to 8, rank columns through the lean kernels (below 24) and the tile
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


# rows that are no whole 16-byte vectors (one bulk copy of the granules that cover a tile, edge elements one per lane): every
# misalignment, register-resident and streamed widths, the causal form, tensors that start off a 16-byte boundary
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(64, 17), (70, 63), (333, 257), (130, 777), (90, 1023), (66, 2049), (3, 777), (64, 5001)])
@pytest.mark.parametrize("shift", [0, 3])
def test_softmax_ragged_rows(cuda_device, dtype, rows, D, shift):
    from metal_candle_b200 import backend as B

    def put(a):   # the values of `a` in a tensor that starts `shift` elements into an allocation
        buf = torch.full((a.size + shift + 8,), float("nan"), dtype=dtype, device=cuda_device)
        view = buf[shift:shift + a.size].view(a.shape)
        view.copy_(torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device).to(dtype))
        return view, buf

    x, dy = rounded(S.normal(41, "x", (rows, D)) * 3, dtype), rounded(S.normal(41, "dy", (rows, D)), dtype)
    (xt, _), (dyt, _), (yt, ybuf), (dxt, dxbuf) = put(x), put(dy), put(x * 0), put(x * 0)
    want = R.softmax_stable(x.astype(np.float64))
    B.softmax_fused(xt, out=yt)
    assert R.max_abs_normalised(back(yt), want) <= TOL[dtype]
    B.softmax_backward(yt, dyt, out=dxt)
    y = back(yt).astype(np.float64)
    assert R.max_abs_normalised(back(dxt), y * (dy - (dy * y).sum(-1, keepdims=True))) <= TOL[dtype]
    for buf in (ybuf, dxbuf):   # nothing outside the rows was written
        assert torch.isnan(buf[:shift]).all() and torch.isnan(buf[shift + rows * D:]).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("seq", [65, 777, 1031, 2049])
def test_softmax_causal_ragged_rows(cuda_device, dtype, seq):
    from metal_candle_b200 import _lib, backend as B

    x, dy = (rounded(S.normal(42, n, (2, seq, seq)), dtype) for n in ("x", "dy"))
    mask = np.triu(np.full((seq, seq), -np.inf), 1)
    xt, dyt = dev_t(x, dtype, cuda_device), dev_t(dy, dtype, cuda_device)
    y, dx = torch.full_like(xt, float("nan")), torch.full_like(xt, float("nan"))
    lib = _lib.load()
    code, st = B._dtype_code(xt), torch.cuda.current_stream().cuda_stream
    _lib.check(lib.mcb_softmax_causal_fwd(xt.data_ptr(), y.data_ptr(), 2 * seq, seq, seq, 0.5, code, st))
    want = R.softmax_stable(0.5 * x.astype(np.float64) + mask)
    assert R.max_abs_normalised(back(y), want) <= TOL[dtype]
    _lib.check(lib.mcb_softmax_causal_bwd(y.data_ptr(), dyt.data_ptr(), dx.data_ptr(), 2 * seq, seq, seq, 0.5, code, st))
    yf = back(y).astype(np.float64)
    assert R.max_abs_normalised(back(dx), 0.5 * yf * (dy - (dy * yf).sum(-1, keepdims=True))) <= TOL[dtype]
    assert np.all(back(dx)[:, np.triu_indices(seq, 1)[0], np.triu_indices(seq, 1)[1]] == 0)


# the loss: short rows (block kernel), rows over 1, 2 (32000 bfloat16), 4 (32000 float32) and 8 CTAs, rows that are no whole
# vectors, more rows than clusters, ignored targets, int32 and int64 targets
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,V,tdtype", [(5, 50, torch.int64), (3, 8192, torch.int32), (700, 8193, torch.int64), (30, 32000, torch.int32), (90, 50257, torch.int32),
                                           (160, 60001, torch.int64), (40, 151936, torch.int64)])
def test_cross_entropy_rows(cuda_device, dtype, rows, V, tdtype):
    from metal_candle_b200 import _lib
    from metal_candle_b200.training import cross_entropy_loss

    x = rounded(S.normal(43, "x", (1, rows, V)) * 2, dtype)
    t = np.random.default_rng(7).integers(0, V, (1, rows))
    t[0, 0], t[0, -1], t[0, 1] = 0, V - 1, -1
    if rows > 20:
        t[0, 7:12] = -1
    xt = dev_t(x, dtype, cuda_device)
    before = xt.clone()
    loss, grad = cross_entropy_loss(xt, torch.from_numpy(t).to(cuda_device).to(tdtype), ignore_index=-1, return_grad=True)
    assert torch.equal(xt, before)
    x64 = x[0].astype(np.float64)
    lse = np.log(np.exp(x64 - x64.max(-1, keepdims=True)).sum(-1)) + x64.max(-1)
    keep = t[0] >= 0
    nll = lse[keep] - x64[keep, t[0][keep]]
    assert abs(float(loss) - nll.mean()) <= 1e-5 * abs(nll.mean())   # float32 sums of exponentials of 2^-22 each
    want = np.where(keep[:, None], np.exp(x64 - lse[:, None]), 0.0)
    want[np.nonzero(keep)[0], t[0][keep]] -= 1.0
    assert R.max_abs_normalised(back(grad)[0], want / keep.sum()) <= TOL[dtype]
    # the in-place form of the training step
    tg = torch.from_numpy(t[0].astype(np.int32)).to(cuda_device)
    nl, cnt, ls = torch.empty(rows, device=cuda_device), torch.empty(1, dtype=torch.int32, device=cuda_device), torch.empty(2, device=cuda_device)
    _lib.check(_lib.load().mcb_cross_entropy(xt.data_ptr(), tg.data_ptr(), nl.data_ptr(), cnt.data_ptr(), ls.data_ptr(), rows, V, 1,
                                             0 if dtype == torch.float32 else 1, torch.cuda.current_stream().cuda_stream))
    assert R.max_abs_normalised(back(xt), want / keep.sum()) <= TOL[dtype] and int(cnt) == int(keep.sum())
    assert abs(float(ls[0]) - nll.mean()) <= 1e-5 * abs(nll.mean())
    assert _lib.device_status() == 0


# logits and gradient that start off a 16-byte boundary: by the same amount (the cluster kernel, elements in front of the
# first whole vector), by different ones (the block kernel); what surrounds the gradient is not written
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [8193, 32000, 50257])
@pytest.mark.parametrize("shift,out_shift", [(0, 0), (1, 1), (3, 3), (3, 0), (1, 2)])
def test_cross_entropy_of_shifted_rows(cuda_device, dtype, V, shift, out_shift):
    from metal_candle_b200 import _lib, backend as B

    rows = 7
    x = rounded(S.normal(44, "x", (rows, V)) * 2, dtype)
    t = torch.tensor([0, V - 1, -1, 5, V // 2, 1, V - 2], device=cuda_device)
    buf = torch.full((rows * V + shift + 8,), 100.0, dtype=dtype, device=cuda_device)   # a neighbour would win every maximum
    buf[shift:shift + rows * V] = torch.from_numpy(np.ascontiguousarray(x)).to(cuda_device).to(dtype).view(-1)
    out = torch.full((rows * V + out_shift + 8,), float("nan"), dtype=dtype, device=cuda_device)
    t32, info = (torch.empty(n, dtype=torch.int32, device=cuda_device) for n in (rows, 3))
    nll, loss = (torch.empty(n, device=cuda_device) for n in (rows, 2))
    e = buf.element_size()
    _lib.check(_lib.load().mcb_cross_entropy_out(buf.data_ptr() + shift * e, out.data_ptr() + out_shift * e, t.data_ptr(), 8, 0, 0, t32.data_ptr(),
                                                 info.data_ptr(), None, None, nll.data_ptr(), loss.data_ptr(), rows, V,
                                                 B._dtype_code(buf), B._stream()))
    x64 = x.astype(np.float64)
    p = np.exp(x64 - x64.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    keep, at = (t >= 0).cpu().numpy(), np.maximum(t.cpu().numpy(), 0)
    want_nll = np.where(keep, -np.log(p[np.arange(rows), at]), 0.0)
    p[np.arange(rows), at] -= 1.0
    got = out[out_shift:out_shift + rows * V].view(rows, V)
    assert np.abs(back(nll) - want_nll).max() <= 1e-5 * np.abs(want_nll).max()
    assert abs(float(loss[0]) - want_nll.sum() / keep.sum()) <= 1e-5 * want_nll.mean()
    assert R.max_abs_normalised(back(got), np.where(keep[:, None], p, 0.0) / keep.sum()) <= TOL[dtype]
    assert torch.isnan(out[:out_shift]).all() and torch.isnan(out[out_shift + rows * V:]).all()
    assert _lib.device_status() == 0


# few tokens: tiles of 32 to 256 columns, reductions in 1, 2, 4 and 8 parts (a part of one k-block included), ragged rows,
# columns and reductions, rank columns with and without, bias and residual; and the first shapes past the rule
@pytest.mark.parametrize("M,K,N,r", [(1, 8, 8, 0), (5, 64, 32, 8), (130, 136, 264, 16), (333, 4864, 896, 8), (512, 20000, 896, 0),
                                     (64, 1024, 40, 33), (257, 896, 1152, 48), (1000, 896, 896, 16), (1100, 4864, 256, 32),
                                     (2048, 2048, 128, 64), (1024, 1000, 4864, 0), (1280, 896, 4864, 8)])
def test_bf16_linear_few_tiles(cuda_device, M, K, N, r):
    from metal_candle_b200 import _lib, backend as B

    c = {k: S.bf16_round(v) for k, v in S.lora_linear_case(51, M, K, N, max(r, 1)).items()}
    res, dres, bias = (S.bf16_round(S.normal(51, n, s)) for n, s in (("res", (M, N)), ("dres", (M, K)), ("bias", (N,))))
    bf = torch.bfloat16
    x, W, dy, rt, drt, bt = (dev_t(a, bf, cuda_device) for a in (c["x"], c["W"], c["dy"], res, dres, bias))
    A, Bm = (dev_t(c[k], torch.float32, cuda_device) if r else None for k in ("A", "B"))
    y, h = B.lora_linear_forward(x, W, bt, A, Bm, 2.0, residual=rt)
    dx, dA, dB = B.lora_linear_backward(x, B.transpose_2d(W), A, Bm, 2.0, dy, h_save=h, dx_residual=drt)
    if r:
        want_y, want_h = R.lora_linear_forward(c["x"], c["W"], bias, c["A"], c["B"], 2.0)
        wdx, wdA, wdB = R.lora_linear_backward(c["x"], c["W"], c["A"], c["B"], 2.0, c["dy"])
        assert R.max_abs_normalised(back(h)[:r, :M].T, 2.0 * want_h) <= 2e-2
        assert R.max_abs_normalised(back(dA), wdA) <= 2e-2 and R.max_abs_normalised(back(dB), wdB) <= 2e-2
    else:
        want_y = R.linear(c["x"], c["W"]) + bias
        wdx = c["dy"].astype(np.float64) @ c["W"].astype(np.float64)
    assert R.max_abs_normalised(back(y), want_y + res) <= 2e-2
    assert R.max_abs_normalised(back(dx), wdx + dres) <= 2e-2
    assert _lib.device_status() == 0


@pytest.mark.parametrize("M,K,F", [(1, 64, 128), (129, 904, 256), (333, 896, 4864), (512, 128, 4736), (513, 128, 4864)])
def test_gate_up_swiglu_few_tokens(cuda_device, M, K, F):
    from metal_candle_b200 import backend as B

    x, wg, wu = (S.bf16_round(S.normal(52, n, s) / (1 if n == "x" else K ** 0.5)) for n, s in (("x", (M, K)), ("g", (F, K)), ("u", (F, K))))
    xt, gt, ut = (dev_t(a, torch.bfloat16, cuda_device) for a in (x, wg, wu))
    gate, up, act = B.linear_swiglu_forward(xt, B.interleave_gate_up(gt, ut))
    g, u = (x.astype(np.float64) @ w.astype(np.float64).T for w in (wg, wu))
    for got, want in ((gate, g), (up, u), (act, g / (1 + np.exp(-g)) * u)):
        assert R.max_abs_normalised(back(got), want) <= 2e-2


# key blocks x kv heads from one to more than the SMs: 1, 4, 8, 2 and 1 CTAs share a key block, 4 and 8 in the last two, whose
# last key block has 2 and 4 query steps, so that some of its CTAs have none
@pytest.mark.parametrize("nb,G,seq", [(1, 1, 128), (1, 7, 128), (4, 7, 256), (16, 3, 512), (40, 2, 512), (1, 1, 1024), (1, 2, 1024)])
def test_attention_backward_shared_key_blocks(cuda_device, nb, G, seq):
    from metal_candle_b200 import backend as B

    q, k, v, do = (S.bf16_round(S.normal(92, n, s)) for n, s in (("q", (nb, G, seq, 64)), ("k", (nb, seq, 64)), ("v", (nb, seq, 64)),
                                                                 ("do", (nb, G, seq, 64))))
    bf = torch.bfloat16
    qd, dod = (dev_t(t.reshape(nb, G * seq, 64), bf, cuda_device) for t in (q, do))
    kd, vd = dev_t(k, bf, cuda_device), dev_t(v, bf, cuda_device)
    o, lse = B.attention_causal_forward(qd, kd, vd, G, 0.125)
    first = B.attention_causal_backward(qd, kd, vd, o, lse, dod, G, 0.125)
    again = B.attention_causal_backward(qd, kd, vd, o, lse, dod, G, 0.125)
    for got, rep, want in zip(first, again, R.causal_gqa_attention_backward(q, k, v, 0.125, do)):
        assert torch.equal(got, rep)
        assert np.abs(back(got).reshape(want.shape) - want).max() <= 2e-2 * np.abs(want).max()


# nb kv heads, G query heads each, S positions: one row, the edges of the 64-key blocks and 128-query tiles, remainders; in
# the last two, 4 CTAs share a key block and the last one has a single query step
RAGGED_ATTENTION = [(1, 1, 1), (2, 3, 5), (1, 7, 63), (2, 1, 64), (2, 7, 65), (4, 2, 111), (2, 1, 127), (1, 2, 129), (2, 2, 193), (1, 7, 333),
                    (1, 1, 897), (2, 1, 700)]


@pytest.mark.parametrize("nb,G,seq", RAGGED_ATTENTION)
@pytest.mark.parametrize("token_major", [False, True])
def test_attention_of_any_length(cuda_device, nb, G, seq, token_major):
    from metal_candle_b200 import _lib, backend as B

    q, k, v, do = (S.bf16_round(S.normal(91, n, s)) for n, s in (("q", (nb, G, seq, 64)), ("k", (nb, seq, 64)), ("v", (nb, seq, 64)),
                                                                 ("do", (nb, G, seq, 64))))
    want_o, want_lse, _ = R.causal_gqa_attention(q, k, v, 0.125)
    wdq, wdk, wdv = R.causal_gqa_attention_backward(q, k, v, 0.125, do)
    kvh = nb if token_major else 0

    def layout(a):   # one batch of nb kv heads: [nb, G, S, d] -> [S, nb * G * d]
        return a.transpose(2, 0, 1, 3).reshape(seq, nb * G * 64) if token_major else a.reshape(nb, G * seq, 64)

    bf = torch.bfloat16
    qd, kd, vd = dev_t(q.reshape(nb, G * seq, 64), bf, cuda_device), dev_t(k, bf, cuda_device), dev_t(v, bf, cuda_device)
    o, lse = B.attention_causal_ragged_forward(qd, kd, vd, G, 0.125, kv_heads=kvh)
    dq, dk, dv = B.attention_causal_ragged_backward(qd, kd, vd, o, lse, dev_t(layout(do), bf, cuda_device), G, 0.125, kv_heads=kvh)
    assert _lib.device_status() == 0
    assert np.abs(back(lse).reshape(nb, G, seq) - want_lse).max() <= 2e-2
    # one position attends to itself alone: P = 1 and dS = 0, so dq and dk are the rounding of dP - delta around zero
    # (a sum of 64 products of size 1 in float32, times |k| / 8: below 1e-4)
    floor = 1e-2 if seq == 1 else 0.0
    for got, want in ((o, layout(want_o)), (dq, wdq.reshape(nb, G * seq, 64)), (dk, wdk), (dv, wdv)):
        assert np.abs(back(got) - want).max() <= 2e-2 * max(np.abs(want).max(), floor)


def test_attention_of_any_length_reads_no_other_head(cuda_device):
    """Tiles that reach past the end of a sequence: what lies there (the next head, inf and NaN in it) must not matter."""
    from metal_candle_b200 import backend as B

    seq, G = 77, 2
    g = torch.Generator(device=cuda_device).manual_seed(3)
    q, k, v, do = (torch.randn(3, rows, 64, device=cuda_device, generator=g).to(torch.bfloat16) for rows in (G * seq, seq, seq, G * seq))
    alone = [t[:1].contiguous() for t in (q, k, v, do)]
    for t, bad in ((q, float("nan")), (k, float("inf")), (v, float("nan")), (do, float("inf"))):
        t[1:] = bad

    def run(q, k, v, do):
        o, lse = B.attention_causal_ragged_forward(q, k, v, G, 0.125)
        return (o, lse) + B.attention_causal_ragged_backward(q, k, v, o, lse, do, G, 0.125)

    # the number of CTAs that share a key block depends on the number of heads, so sums may be ordered differently
    for a, b in zip(run(*alone), run(q, k, v, do)):
        assert torch.isfinite(b[0].float()).all()
        torch.testing.assert_close(a[0].float(), b[0].float(), rtol=2e-2, atol=1e-3)


# tokens of one share of the heads per block (many) and of several, down to one head each (few)
@pytest.mark.parametrize("batch,seq", [(1, 1), (3, 111), (2, 1500), (1, 20000)])
@pytest.mark.parametrize("inverse", [0, 1])
def test_rope_qkv_shares_heads(cuda_device, batch, seq, inverse):
    """The merged launch against the three single ones, whose results it has to repeat to the bit."""
    from metal_candle_b200 import _lib
    from metal_candle_b200.backend import MCB_BF16, _ptr, _stream

    lib = _lib.init(0)
    g = torch.Generator(device=cuda_device).manual_seed(5)
    heads, width = (14, 2, 2), 18 * 64
    fused = torch.randn(batch * seq, width, device=cuda_device, generator=g).to(torch.bfloat16)
    major = [torch.randn(batch, h, seq, 64, device=cuda_device, generator=g).to(torch.bfloat16) for h in heads]
    want_fused, want_major = fused.clone(), [m.clone() for m in major]
    _lib.check(lib.mcb_rope_relayout_qkv(_ptr(fused), *(_ptr(m) for m in major), batch, seq, 14, 2, 64, 1e6, inverse, width, MCB_BF16, _stream()))
    at = 0
    for m, h, rotate in zip(want_major, heads, (1, 1, 0)):
        src, dst = (m, want_fused) if inverse else (want_fused, m)
        _lib.check(lib.mcb_rope_relayout_ex(_ptr(src), _ptr(dst), batch, seq, h, 64, 1e6, rotate, inverse, width, at, MCB_BF16, _stream()))
        at += h * 64
    assert torch.equal(fused, want_fused) and all(torch.equal(a, b) for a, b in zip(major, want_major))


@pytest.mark.parametrize("count", [1, 64, 65, 256, 257, 600])
def test_adamw_many_tensors(cuda_device, count):
    """One launch holds 64 or 256 descriptors; the update itself is elementwise, so it equals that of one tensor at a time."""
    from metal_candle_b200.training import AdamW, AdamWConfig

    g = torch.Generator(device=cuda_device).manual_seed(9)
    sizes = [1 + (37 * i) % 203 for i in range(count)]
    together = [torch.randn(n, device=cuda_device, generator=g) for n in sizes]
    grads = [torch.randn(n, device=cuda_device, generator=g) for n in sizes]
    single = [p.clone() for p in together]
    a, b = AdamW(AdamWConfig()), AdamW(AdamWConfig())
    for _ in range(2):
        a.step_vars(together, grads)
        for p, gr in zip(single, grads):
            b.step_var(p, gr)
    assert a.step_count == b.step_count == 2 * count
    assert all(torch.equal(p, q) for p, q in zip(together, single))


@pytest.mark.parametrize("count", [2, 70, 200, 300])
def test_adamw_of_overlapping_tensors(cuda_device, count):
    """A parameter listed twice, and a buffer next to views of it: the update is that of one tensor after the other."""
    from metal_candle_b200.training import AdamW, AdamWConfig

    def lists(seed):
        g = torch.Generator(device=cuda_device).manual_seed(seed)
        flat = torch.randn(5000, device=cuda_device, generator=g)
        others = [torch.randn(1000 + i, device=cuda_device, generator=g) for i in range(count - 2)]
        variables = [flat[100:3000]] + others + [flat]
        variables[count // 2:count // 2] = [flat[100:3000], flat[:200]]
        return flat, variables, [torch.randn(v.shape, device=cuda_device, generator=g) for v in variables]

    (flat_a, vars_a, grads), (flat_b, vars_b, _) = lists(1), lists(1)
    a, b = AdamW(AdamWConfig()), AdamW(AdamWConfig())
    for _ in range(3):
        a.step_vars(vars_a, grads)
        for p, gr in zip(vars_b, grads):
            b.step_var(p, gr)
    assert torch.equal(flat_a, flat_b) and all(torch.equal(p, q) for p, q in zip(vars_a, vars_b))


def test_loss_grid_does_not_depend_on_earlier_vocabularies(cuda_device, tmp_path):
    """Two vocabularies whose rows take the same number of CTAs but other amounts of shared memory: the grid of either is the
    same whichever a process meets first."""
    import json
    import subprocess
    import sys
    from pathlib import Path

    child = """
import json, sys
import torch
from torch.profiler import ProfilerActivity, profile
from metal_candle_b200.training import cross_entropy_loss
t = torch.zeros(1, 400, dtype=torch.int64, device="cuda")
vocabularies = [int(v) for v in sys.argv[2:]]
for v in vocabularies:
    cross_entropy_loss(torch.zeros(1, 400, v, device="cuda"), t, return_grad=True)
grids = {}
for v in vocabularies:
    x = torch.zeros(1, 400, v, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        cross_entropy_loss(x, t, return_grad=True)
        torch.cuda.synchronize()
    p.export_chrome_trace(sys.argv[1])
    grids[v] = [e["args"]["grid"] for e in json.load(open(sys.argv[1]))["traceEvents"] if "cluster_kernel" in e.get("name", "")]
print(json.dumps(grids))
"""
    runs = []
    for order in (("50257", "151936"), ("151936", "50257")):
        r = subprocess.run([sys.executable, "-c", child, str(tmp_path / "trace.json"), *order], capture_output=True, text=True,
                           cwd=Path(__file__).resolve().parent.parent, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        runs.append(json.loads(r.stdout.splitlines()[-1]))
    if not all(runs[0].values()):
        pytest.skip("no kernel records from the profiler")
    assert runs[0] == runs[1]
    assert runs[0]["50257"] != runs[0]["151936"]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M", [1, 64, 1000])
@pytest.mark.parametrize("K,N", [(1 << 31, 64), (64, 1 << 31), ((1 << 32) - 8, 64)])
def test_lora_refuses_dimensions_beyond_31_bits(cuda_device, dtype, M, K, N):
    """The kernels count in 32 bits; the ABI admits dimensions of u32.  (The buffers are small: nothing may be launched.)"""
    from metal_candle_b200 import _lib, backend as B

    small = torch.empty(1 << 20, dtype=torch.uint8, device=cuda_device)
    at = small.data_ptr() + (-small.data_ptr()) % 1024
    lib, code = _lib.load(), B._dtype_code(torch.empty(0, dtype=dtype))
    before = lib.mcb_launch_count()
    calls = (lambda: lib.mcb_lora_delta_fwd(at, at, at, at, M, K, N, 8, 2.0, code, at, 1 << 62, B._stream()),
             lambda: lib.mcb_lora_linear_fwd(at, at, None, at, at, at, at, M, K, N, 8, 2.0, code, 0, at, 1 << 62, B._stream()))
    for call in calls:
        assert call() == -2 and b"2^31" in lib.mcb_last_error() and lib.mcb_launch_count() == before


@pytest.mark.parametrize("M", [1, 5, 256, 257])
def test_bf16_delta_is_recorded_by_the_profile(cuda_device, M):
    """Both forms of the delta (one cluster launch up to 256 tokens, the GEMM beyond) report to the per-kernel profile."""
    from metal_candle_b200 import _lib, backend as B

    K, N, r = 512, 384, 8
    x = torch.zeros(M, K, dtype=torch.bfloat16, device=cuda_device)
    A, Bm = torch.zeros(K, r, device=cuda_device), torch.zeros(r, N, device=cuda_device)
    _lib.profile_enable(True)
    try:
        _lib.profile_summary(2)
        B.lora_forward_fused(x, A, Bm, 2.0)
        launches, ms, flops, _ = _lib.profile_summary(2)
    finally:
        _lib.profile_enable(False)
    assert launches == 1 and ms > 0 and flops == 2.0 * M * r * (K + N)


# float32 products on the tensor cores: rows and indices around the 128 x 128 (64) tile and the 64-index step, the last reduction
# of the short kernel (64) and the first beyond, both orders of either operand, reductions shared by 1 to 8 CTAs
@pytest.mark.parametrize("M,K,N", [(128, 64, 128), (129, 65, 129), (127, 128, 64), (1, 127, 1), (300, 1024, 65), (1200, 200, 1100)])
def test_f32_product_rounds_like_float32(cuda_device, M, K, N):
    """Against float64, relative to the sum of magnitudes: a float32 sum of K terms, whatever its order, errs by up to K 2^-24;
    what the parts' products leave out is at most 2^-20 of each product, the worst for any of them and not for their sum."""
    from metal_candle_b200 import backend as B
    from metal_candle_b200._lib import MCB_W_OUT_IN

    g = torch.Generator(device=cuda_device).manual_seed(M + K)
    x, w, dy = (torch.randn(*s, device=cuda_device, generator=g) for s in ((M, K), (N, K), (M, N)))
    wt = w.t().contiguous()
    bound = 2.0 ** -20
    for got, p, q in ((B.lora_linear_forward(x, w, None, None, None, 1.0)[0], x, w.t()), (B.matmul(x, wt), x, w.t()),
                      (B.lora_linear_backward(None, wt, None, None, 1.0, dy)[0], dy, w),
                      (B.lora_linear_backward(None, w, None, None, 1.0, dy, weight_layout=MCB_W_OUT_IN)[0], dy, w)):
        err = (got.double() - p.double() @ q.double()).abs() / (p.double().abs() @ q.double().abs())
        assert err.max().item() <= bound


# operands of one sign and of both: what is left out of a product or cut off a sum must not add up
@pytest.mark.parametrize("M,K,N", [(512, 768, 768), (300, 65, 200), (257, 1024, 129), (300, 1000, 64)])
@pytest.mark.parametrize("values", ["normal", "uniform01", "uniform12", "shifted"])
def test_f32_product_error_has_no_sign(cuda_device, values, M, K, N):
    """Against float64.  A float32 result is rounded to 2^-24 of itself; sums of rounded terms wander about it, so the error of the
    whole result stays below one unit in the last place, 2^-23, and its mean below half of one."""
    from metal_candle_b200 import backend as B
    from metal_candle_b200._lib import MCB_W_OUT_IN

    g = torch.Generator(device=cuda_device).manual_seed(M * N + K)
    make = {"normal": lambda *s: torch.randn(*s, device=cuda_device, generator=g), "uniform01": lambda *s: torch.rand(*s, device=cuda_device, generator=g),
            "uniform12": lambda *s: torch.rand(*s, device=cuda_device, generator=g) + 1.0,
            "shifted": lambda *s: torch.randn(*s, device=cuda_device, generator=g) + 3.0}[values]
    x, w, dy = make(M, K), make(N, K), make(M, N)
    wt = w.t().contiguous()
    for got, p, q in ((B.lora_linear_forward(x, w, None, None, None, 1.0)[0], x, w.t()), (B.matmul(x, wt), x, w.t()),
                      (B.lora_linear_backward(None, w, None, None, 1.0, dy, weight_layout=MCB_W_OUT_IN)[0], dy, w)):
        want = p.double() @ q.double()
        err = got.double() - want
        assert (err.norm() / want.norm()).item() <= 2.0 ** -23
        assert abs((err.sum() / want.abs().sum()).item()) <= 2.0 ** -24


def test_f32_product_of_equal_operands_keeps_every_bit(cuda_device):
    """x = 1 + 2^-7 - 2^-23: products whose smaller parts are as large as they get.  A row of one such term is the product rounded once
    (2^-24), one of K terms a sum of K / 16 + 1 roundings."""
    from metal_candle_b200 import backend as B

    v = 1.0 + 2.0 ** -7 - 2.0 ** -23
    for K, terms in ((128, 1), (128, 128), (1024, 1024)):
        x, w = torch.zeros(130, K, device=cuda_device), torch.zeros(70, K, device=cuda_device)
        x[:, :terms] = v
        w[:, :terms] = -v
        y = B.lora_linear_forward(x, w, None, None, None, 1.0)[0].double()
        want = -terms * v * v
        assert ((y - want).abs().max().item()) <= abs(want) * 2.0 ** -24 * (1 if terms == 1 else terms // 16 + 1)


# short reductions: the first and the last of the short kernel, the first of the tile kernel behind it; widths with and without whole
# 16-byte stores, rows beyond a block of 64
@pytest.mark.parametrize("M,K,N,r", [(1, 1, 1, 1), (65, 5, 63, 3), (64, 31, 64, 8), (130, 32, 132, 32), (200, 32, 66, 16), (97, 33, 130, 30)])
def test_f32_short_reduction_edges(cuda_device, M, K, N, r):
    """With bias, residual and adapter, against float64: a chain of n float32 operations errs by at most n 2^-24 of the sum of
    magnitudes; the adapter's h has K + 1 of its own, and an output K + r + 4."""
    from metal_candle_b200 import backend as B
    from metal_candle_b200._lib import MCB_W_OUT_IN

    g = torch.Generator(device=cuda_device).manual_seed(M * K + N)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g)  # noqa: E731
    x, w, bias, a, b, res, dy = rnd(M, K), rnd(N, K), rnd(N), rnd(K, r), rnd(r, N), rnd(M, N), rnd(M, N)
    d = lambda t: t.double()  # noqa: E731
    got = B.lora_linear_forward(x, w, bias, a, b, 2.0, residual=res)[0]
    want = d(x) @ d(w).t() + d(bias) + 2 * (d(x) @ d(a)) @ d(b) + d(res)
    size = d(x).abs() @ d(w).abs().t() + d(bias).abs() + 2 * (d(x).abs() @ d(a).abs()) @ d(b).abs() + d(res).abs()
    assert ((d(got) - want).abs() <= size * 2.0 ** -24 * (2 * K + r + 5)).all()
    for wt, kw in ((w.t().contiguous(), {}), (w, dict(weight_layout=MCB_W_OUT_IN))):
        dx = rnd(M, K)
        got = B.lora_linear_backward(x, wt, a, b, 2.0, dy, dx_residual=dx, **kw)[0]
        want = d(dy) @ d(w) + 2 * (d(dy) @ d(b).t()) @ d(a).t() + d(dx)
        size = d(dy).abs() @ d(w).abs() + 2 * (d(dy).abs() @ d(b).abs().t()) @ d(a).abs().t() + d(dx).abs()
        assert ((d(got) - want).abs() <= size * 2.0 ** -24 * (2 * N + r + 5)).all()
    got = B.matmul(x, w.t().contiguous())
    assert ((d(got) - d(x) @ d(w).t()).abs() <= d(x).abs() @ d(w).abs().t() * 2.0 ** -24 * (K + 1)).all()


def test_f32_product_of_extreme_values(cuda_device):
    """Infinities, NaN, the largest and the smallest numbers come out as float32 arithmetic has them (each output is one product:
    one term per row is not zero)."""
    from metal_candle_b200 import backend as B

    K = 200
    a = torch.tensor([3.4e38, -3.4e38, 1e31, 1e38, 1.2e-38, 1e-38, 3e-42, 1e-45, 0.0, 1.7, -2.3e-20, float("inf"), float("nan")], device=cuda_device)
    b = torch.tensor([1.0, -0.25, 3.3e-39, 1e-30, 1e25, 3.4e38, 1e-3], device=cuda_device)
    x = torch.zeros(len(a), K, device=cuda_device)
    x[:, 77] = a
    w = torch.zeros(len(b), K, device=cuda_device)
    w[:, 77] = b
    y, _ = B.lora_linear_forward(x, w, None, None, None, 1.0)
    want = (a.double()[:, None] * b.double()[None, :]).float()
    assert torch.equal(y.isnan(), want.isnan())
    ok = ~want.isnan()
    # the products of the smaller parts that are left out (2^-20), and the spacing of the smallest numbers
    assert torch.equal(y[ok].isinf(), want[ok].isinf())
    fin = ok & want.isfinite()
    assert ((y[fin].double() - want[fin].double()).abs() <= want[fin].double().abs() * 2.0 ** -20 + 2.0 ** -149).all()


# outputs that the parts spoil, among others: whole tiles and ragged ones, reductions of one CTA and shared by up to 8, 64-wide tiles
@pytest.mark.parametrize("M,K,N,r", [(512, 768, 768, 8), (300, 200, 132, 40), (257, 1024, 63, 3), (1200, 100, 1101, 16)])
def test_f32_outputs_that_are_computed_again(cuda_device, M, K, N, r):
    """A NaN, an infinity and a number too large for the parts in x and W touch their rows and columns and nothing else: the other
    outputs keep their bits, those of the large numbers are a float32 chain of FMAs (its error: a unit per term of the magnitudes)."""
    from metal_candle_b200 import backend as B

    g = torch.Generator(device=cuda_device).manual_seed(M + N)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g)  # noqa: E731
    x, w, bias, a, b, res = rnd(M, K), rnd(N, K), rnd(N), rnd(K, r), rnd(r, N), rnd(M, N)
    clean = B.lora_linear_forward(x, w, bias, a, b, 2.0, residual=res)[0]
    xs, ws = x.clone(), w.clone()
    xs[1, 3], xs[M // 2, K - 1], xs[M - 1, 0] = float("nan"), float("inf"), 3e33
    ws[2, 5], ws[N - 1, K // 2] = float("nan"), -2e34
    got = B.lora_linear_forward(xs, ws, bias, a, b, 2.0, residual=res)[0]
    rows, cols = [1, M // 2, M - 1], [2, N - 1]
    kept = torch.ones(M, N, dtype=torch.bool, device=cuda_device)
    kept[rows] = False
    kept[:, cols] = False
    assert torch.equal(got[kept], clean[kept])
    want = xs.double() @ ws.double().t() + bias.double() + 2 * (xs.double() @ a.double()) @ b.double() + res.double()
    size = xs.double().abs() @ ws.double().abs().t() + bias.double().abs() + 2 * (xs.double().abs() @ a.double().abs()) @ b.double().abs() + res.double().abs()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    fin = want.isfinite() & ~kept
    assert ((got.double() - want)[fin].abs() <= size[fin] * 2.0 ** -24 * (2 * K + r + 5)).all()
    # gradients that are added to what is there, an infinity among the terms (rank 24: products of the tile kernel)
    a, b, dy = rnd(K, 24), rnd(24, N), rnd(M, N)
    xs = x.clone()
    xs[M // 2, 1] = float("inf")
    start = rnd(K, 24)
    grads = [start.clone(), rnd(24, N)]
    B.lora_linear_backward(xs, w.t().contiguous(), a, b, 1.0, dy, grad_a=grads[0], grad_b=grads[1], accumulate=True)
    h = dy.double() @ b.double().t()
    want = start.double() + xs.double().t() @ h
    size = start.double().abs() + x.double().abs().t() @ (dy.double().abs() @ b.double().abs().t())
    assert torch.equal(grads[0].isinf(), want.isinf())
    ok = want.isfinite()
    assert ((grads[0].double() - want)[ok].abs() <= size[ok] * 2.0 ** -24 * (M + N + 3)).all()


def test_f32_product_of_nan_costs_no_multiple(cuda_device):
    """A run that has diverged goes on at the pace of float32 FMAs, not at that of a serial sum per output (86 times the clean call
    where that was done): eight times the clean call at most."""
    from metal_candle_b200 import backend as B

    def us(x, w):
        best = float("inf")
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            B.lora_linear_forward(x, w, None, None, None, 1.0)
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    x, w = torch.randn(2048, 1536, device=cuda_device), torch.randn(1536, 1536, device=cuda_device)
    clean = us(x, w)
    assert us(torch.full_like(x, float("nan")), w) <= 8 * clean


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("seq", [32, 64, 255, 256, 512, 777, 1024, 1100])
def test_causal_softmax_backward_in_registers(cuda_device, dtype, seq):
    """One to eight vectors per lane, whole and ragged rows: exact zeros behind the query position, against the oracle."""
    from metal_candle_b200 import _lib
    from metal_candle_b200.backend import _dtype_code, _ptr, _stream

    rng = np.random.default_rng(seq)
    rows = 3 * seq
    y = rng.random((rows, seq))
    y[np.arange(seq)[None, :] > (np.arange(rows) % seq)[:, None]] = 0.0
    y, dy = rounded(y / y.sum(1, keepdims=True), dtype), rounded(rng.standard_normal((rows, seq)), dtype)
    yd, dyd = dev_t(y, dtype, cuda_device), dev_t(dy, dtype, cuda_device)
    dx = torch.full_like(yd, 7.0)
    lib = _lib.load()
    _lib.check(lib.mcb_softmax_causal_bwd(_ptr(yd), _ptr(dyd), _ptr(dx), rows, seq, seq, 0.125, _dtype_code(yd), _stream()))
    y64, dy64 = y.astype(np.float64), dy.astype(np.float64)
    want = y64 * (dy64 - (y64 * dy64).sum(1, keepdims=True)) * 0.125
    got = back(dx)
    assert R.max_abs_normalised(got, want) <= TOL[dtype]
    assert (got[np.arange(seq)[None, :] > (np.arange(rows) % seq)[:, None]] == 0.0).all()


def _close_bf16(got, want, tol=2e-2):
    assert got.shape == want.shape and bool(got.isfinite().all())
    assert ((got.double() - want).abs().max() / want.abs().max()).item() <= tol


# 256-token tiles of more than 256 columns (18 to 19 row tiles x 2 to 4 wide column tiles fill the 74 CTA pairs once where narrow ones
# need two rounds): widths of 320 to 512, ragged last rows, columns and k-blocks
@pytest.mark.parametrize("M,K,N", [(4865, 2048, 896), (4608, 2040, 2040), (4700, 3000, 1000), (4801, 2504, 1272), (9400, 4864, 896)])
def test_bf16_linear_wide_tiles(cuda_device, M, K, N):
    from metal_candle_b200 import backend as B

    g = torch.Generator(device=cuda_device).manual_seed(M)
    x, w, bias, res = ((torch.randn(*s, device=cuda_device, generator=g) * f).bfloat16() for s, f in (((M, K), 1.0), ((N, K), K ** -0.5), ((N,), 1.0), ((M, N), 1.0)))
    want = x.double() @ w.double().t()
    _close_bf16(B.lora_linear_forward(x, w, None, None, None, 1.0)[0], want)
    _close_bf16(B.lora_linear_forward(x, w, bias, None, None, 1.0, residual=res)[0], want + bias.double() + res.double())


@pytest.mark.parametrize("M,K,F", [(4600, 2048, 1024), (4500, 2504, 1152), (9300, 4096, 896)])
def test_gate_up_swiglu_wide_tiles(cuda_device, M, K, F):
    """An even and an odd number of 128-feature blocks; against float64 of the same bf16 inputs."""
    from metal_candle_b200 import backend as B

    g = torch.Generator(device=cuda_device).manual_seed(M)
    x, wg, wu = ((torch.randn(*s, device=cuda_device, generator=g) * f).bfloat16() for s, f in (((M, K), 1.0), ((F, K), K ** -0.5), ((F, K), K ** -0.5)))
    gate, up, act = B.linear_swiglu_forward(x, B.interleave_gate_up(wg, wu))
    want_g, want_u = x.double() @ wg.double().t(), x.double() @ wu.double().t()
    _close_bf16(gate, want_g)
    _close_bf16(up, want_u)
    _close_bf16(act, torch.nn.functional.silu(want_g) * want_u)


# ranks of one and several 16-column groups; reductions on either side of the pair kernel's line (1536), rows off the tiles
@pytest.mark.parametrize("M,K,N,r", [(4700, 2048, 2048, 64), (5000, 896, 4864, 16), (4100, 1544, 4096, 16), (20000, 896, 896, 64), (3000, 896, 1160, 40)])
def test_bf16_linear_rank_apart(cuda_device, M, K, N, r):
    """Where the rank intermediate gets a launch of its own: forward, saved intermediate and all gradients against float64, with the
    bounds of the other bf16 parity tests."""
    _linear_with_rank_path(cuda_device, M, K, N, r)


# short reductions of 16384 tokens and more on CTA pairs: from 832 features on, ragged last rows, columns and k-blocks
@pytest.mark.parametrize("M,K,N,r", [(16384, 832, 264, 16), (16390, 896, 896, 16), (17001, 1000, 840, 8), (16384, 840, 904, 40)])
def test_bf16_linear_short_reduction_on_pairs(cuda_device, M, K, N, r):
    _linear_with_rank_path(cuda_device, M, K, N, r)


# fewer than 1024 tokens and many outputs: CTA pairs from 148 tiles of 256 x 256 on where the 128-token tiles pair up (two, not three)
@pytest.mark.parametrize("M,K,N", [(130, 72, 148 * 256), (256, 896, 148 * 256 - 248), (257, 200, 148 * 256), (1000, 136, 37 * 256)])
def test_bf16_linear_few_tokens_many_outputs(cuda_device, M, K, N):
    from metal_candle_b200 import backend as B

    g = torch.Generator(device=cuda_device).manual_seed(M)
    x, w, bias = ((torch.randn(*s, device=cuda_device, generator=g) * f).bfloat16() for s, f in (((M, K), 1.0), ((N, K), K ** -0.5), ((N,), 1.0)))
    # one rounding to bf16 of sums whose operands are exact
    _close_bf16(B.lora_linear_forward(x, w, bias, None, None, 1.0)[0], x.double() @ w.double().t() + bias.double(), 2.0 ** -8)


def _linear_with_rank_path(cuda_device, M, K, N, r):
    from metal_candle_b200 import backend as B

    g = torch.Generator(device=cuda_device).manual_seed(M)
    R_ = lambda *s, f=1.0: torch.randn(*s, device=cuda_device, generator=g) * f  # noqa: E731
    x, w, dy = R_(M, K).bfloat16(), R_(N, K, f=K ** -0.5).bfloat16(), R_(M, N).bfloat16()
    a, b = R_(K, r, f=K ** -0.5), R_(r, N, f=0.1)
    y, h = B.lora_linear_forward(x, w, None, a, b, 2.0)
    dx, da, db = B.lora_linear_backward(x, B.transpose_2d(w), a, b, 2.0, dy, h_save=h)
    X, W, D, A, Bm = (t.double() for t in (x, w, dy, a, b))
    H, G = 2.0 * X @ A, 2.0 * D @ Bm.t()
    _close_bf16(y, X @ W.t() + H @ Bm)
    _close_bf16(h[:r, :M].t(), H)
    assert bool((h[r:, :M] == 0).all())
    _close_bf16(dx, D @ W + G @ A.t())
    _close_bf16(da, X.t() @ G)
    _close_bf16(db, H.t() @ D)


@pytest.mark.parametrize("M,K,N,r", [(4096, 896, 896, 16), (1030, 640, 1536, 8), (20000, 896, 128, 16)])
def test_bf16_linear_stores_nothing_that_nobody_reads(cuda_device, M, K, N, r):
    """A call whose rank path stays in its own tiles writes its packed operands into the workspace and nothing else: the rank
    intermediate leaves the kernel only where a launch of its own computes it for the product behind."""
    from metal_candle_b200 import _lib, backend as B

    g = torch.Generator(device=cuda_device).manual_seed(M)
    x, w = (torch.randn(*s, device=cuda_device, generator=g).bfloat16() for s in ((M, K), (N, K)))
    a, b = torch.randn(K, r, device=cuda_device, generator=g), torch.randn(r, N, device=cuda_device, generator=g)
    y = torch.empty(M, N, dtype=torch.bfloat16, device=cuda_device)
    lib, code = _lib.load(), B._dtype_code(x)
    rp = lib.mcb_lora_rank_padded(r)
    h = torch.empty(rp, lib.mcb_lora_h_pitch(M), dtype=torch.bfloat16, device=cuda_device)
    ws = B.aligned_block(cuda_device, lib.mcb_lora_workspace_bytes(M, K, N, r, code)).fill_(0x5a)
    before = lib.mcb_launch_count()
    _lib.check(lib.mcb_lora_linear_fwd(x.data_ptr(), w.data_ptr(), None, a.data_ptr(), b.data_ptr(), y.data_ptr(), h.data_ptr(), M, K, N, r, 2.0,
                                       code, 0, ws.data_ptr(), ws.numel(), B._stream()))
    assert lib.mcb_launch_count() - before == 2   # the pack and the product
    packed = 2 * ((rp * max(K, N) * 2 + 1023) // 1024 * 1024)
    assert (ws[packed:] == 0x5a).all()
    want = x.double() @ w.double().t() + 2 * (x.double() @ a.bfloat16().double()) @ b.bfloat16().double()
    assert ((y.double() - want).abs().max() / want.abs().max()).item() <= 2e-2


@pytest.mark.parametrize("M,K,N,r", [(2048, 4096, 4096, 16), (2048, 1024, 4096, 40), (4096, 896, 896, 16), (512, 896, 896, 8), (16384, 896, 896, 16)])
def test_profile_counts_a_linear_with_an_adapter_once(cuda_device, M, K, N, r):
    """However many launches a call takes (a rank intermediate of its own, wide tiles or pairs behind it; one kernel; parts of the
    reduction), they are recorded as a linear with a rank path, with 2 M N K + 2 M r (K + N) operations between them."""
    from metal_candle_b200 import _lib, backend as B

    x, w = (torch.zeros(*s, dtype=torch.bfloat16, device=cuda_device) for s in ((M, K), (N, K)))
    a, b = torch.zeros(K, r, device=cuda_device), torch.zeros(r, N, device=cuda_device)
    dy = torch.zeros(M, N, dtype=torch.bfloat16, device=cuda_device)
    _lib.profile_enable(True)
    try:
        for kind in range(4):
            _lib.profile_summary(kind)
        B.lora_linear_forward(x, w, None, a, b, 2.0)
        plain, lora = _lib.profile_summary(0), _lib.profile_summary(2)
        assert plain[0] == 0 and lora[0] >= 1 and lora[2] == 2.0 * M * N * K + 2.0 * M * r * (K + N)
        # a backward without an input gradient computes the rank intermediate alone, and the gradients
        h = torch.zeros(_lib.load().mcb_lora_rank_padded(r), _lib.load().mcb_lora_h_pitch(M), dtype=torch.bfloat16, device=cuda_device)
        B.lora_linear_backward(x, w.t().contiguous(), a, b, 2.0, dy, h_save=h, need_dx=False)
        lora, grad = _lib.profile_summary(2), _lib.profile_summary(1)
        assert lora[2] + grad[2] == 2.0 * M * r * N + 2.0 * M * r * (K + N)
    finally:
        _lib.profile_enable(False)


@pytest.mark.parametrize("M,K,N,r", [(1024, 1024, 4096, 16), (4096, 512, 8192, 64)])
def test_raised_pair_option_keeps_linears_in_one_launch(cuda_device, M, K, N, r):
    """MCB_OPT_PAIR_MIN_K above the reduction: no product on CTA pairs behind a launch of its own for the rank intermediate, as by
    default; the results agree to the rounding of either."""
    from metal_candle_b200 import _lib, backend as B

    g = torch.Generator(device=cuda_device).manual_seed(K)
    x, w = (torch.randn(*s, device=cuda_device, generator=g).bfloat16() for s in ((M, K), (N, K)))
    a, b = torch.randn(K, r, device=cuda_device, generator=g), torch.randn(r, N, device=cuda_device, generator=g)
    lib = _lib.load()

    def launches():
        before = lib.mcb_launch_count()
        y = B.lora_linear_forward(x, w, None, a, b, 2.0, save_hidden=False)[0]
        return lib.mcb_launch_count() - before, y

    apart, y = launches()
    assert apart == 3   # the pack, the rank intermediate, the product
    try:
        _lib.check(lib.mcb_set_option(_lib.MCB_OPT_PAIR_MIN_K, 1 << 20))
        n, z = launches()
        assert n == 2
    finally:
        _lib.check(lib.mcb_set_option(_lib.MCB_OPT_PAIR_MIN_K, 1536))
    assert ((y.double() - z.double()).abs().max() / y.double().abs().max()).item() <= 2e-2
