"""GPU: calls on several streams and from several threads, and calls captured by the caller, against the same calls made
one after the other.  Every kernel sums in a fixed order, so the results have to agree to the bit."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def make_work(dev, seed):
    """A linear with adapter, forward and backward, in bfloat16 and float32, and an attention backward: calls whose kernels
    hand each other operands, rank intermediates, partial sums and row statistics in scratch memory."""
    from metal_candle_b200 import backend as B

    g = torch.Generator(device=dev).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g)  # noqa: E731
    M, K, N, r = 384 + 64 * seed, 896, 640, 16
    A, Bm = rnd(K, r) * 0.05, rnd(r, N) * 0.05
    lin = {dt: (rnd(M, K).to(dt), (rnd(N, K) / 30).to(dt), rnd(M, N).to(dt)) for dt in (torch.bfloat16, torch.float32)}
    wt = {dt: B.transpose_2d(t[1]) for dt, t in lin.items()}
    seq, G = 200 + 32 * seed, 3
    q, do = (rnd(2, G * seq, 64).to(torch.bfloat16) for _ in range(2))
    k, v = (rnd(2, seq, 64).to(torch.bfloat16) for _ in range(2))
    o, lse = B.attention_causal_ragged_forward(q, k, v, G, 0.125)

    def run():
        out = []
        for dt, (x, w, dy) in lin.items():
            y, h = B.lora_linear_forward(x, w, None, A, Bm, 2.0)
            out += [y, *B.lora_linear_backward(x, wt[dt], A, Bm, 2.0, dy, h_save=h)]
        return out + list(B.attention_causal_ragged_backward(q, k, v, o, lse, do, G, 0.125))

    return run


def test_two_streams(cuda_device):
    works = [make_work(cuda_device, s) for s in (0, 3)]
    want = [w() for w in works]
    streams = [torch.cuda.Stream() for _ in works]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):   # enqueued in turn, nothing waits
        for i, (w, s) in enumerate(zip(works, streams)):
            with torch.cuda.stream(s):
                got[i].append(w())
    torch.cuda.synchronize()
    for runs, ref in zip(got, want):
        for out in runs:
            assert all(torch.equal(a, b) for a, b in zip(out, ref))


@pytest.mark.parametrize("own_streams", [False, True])
def test_two_threads(cuda_device, own_streams):
    works = [make_work(cuda_device, s) for s in (1, 4)]
    want = [w() for w in works]
    torch.cuda.synchronize()
    wrong = []

    def loop(i):
        torch.cuda.set_device(cuda_device)
        with torch.cuda.stream(torch.cuda.Stream() if own_streams else torch.cuda.default_stream()):
            outs = [works[i]() for _ in range(20)]
            torch.cuda.current_stream().synchronize()
        wrong.extend(i for out in outs if not all(torch.equal(a, b) for a, b in zip(out, want[i])))

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == []


def test_calls_captured_by_the_caller_outlive_the_scratch_buffer(cuda_device):
    """The graph's scratch memory is its own: later calls that need more of it, on any stream, do not disturb a replay."""
    from metal_candle_b200 import backend as B

    work = make_work(cuda_device, 2)
    want = work()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = work()
    big = torch.randn(65536, 1024, device=cuda_device).to(torch.bfloat16)
    B.lora_forward_fused(big, torch.randn(1024, 64, device=cuda_device), torch.randn(64, 1024, device=cuda_device), 2.0)
    junk = [torch.full((1 << 22,), 7.0, device=cuda_device) for _ in range(8)]
    for _ in range(3):
        graph.replay()
        work()            # eager, between replays
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want))
    del junk


def test_chained_launches_change_nothing(cuda_device):
    """Kernels launched while the one before still runs (MCB_OPT_PDL), against launches that wait for it: a chain in which every
    call reads what the last one wrote or writes over what it reads, in eager form and captured."""
    from metal_candle_b200 import _lib, backend as B

    lib = _lib.load()
    g = torch.Generator(device=cuda_device).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g)  # noqa: E731
    M, H, r = 1100, 896, 16
    A, Bm = rnd(H, r) * 0.05, rnd(r, H) * 0.05
    lin = {dt: (rnd(M, H).to(dt), (rnd(H, H) / 30).to(dt), (1 + 0.1 * rnd(H)).to(dt)) for dt in (torch.bfloat16, torch.float32)}
    wt = {dt: B.transpose_2d(t[1]) for dt, t in lin.items()}
    targets = torch.randint(0, H, (M,), device=cuda_device, generator=g, dtype=torch.int32)

    def chain():
        out = []
        for dt, (x, w, gain) in lin.items():
            h, grad_a = x, torch.zeros(H, r, device=cuda_device)
            grad_b = torch.zeros(r, H, device=cuda_device)
            for _ in range(4):
                n = B.rms_norm_fused(h, 1e-6, weight=gain)
                h2, hs = B.lora_linear_forward(n, w, None, A, Bm, 2.0, residual=h)
                p = B.softmax_fused(h2, out=h2)
                p = B.softmax_backward(p, n, out=p)
                dx, _, _ = B.lora_linear_backward(n, wt[dt], A, Bm, 2.0, p, h_save=hs, grad_a=grad_a, grad_b=grad_b, accumulate=True)
                h, dw = B.rms_norm_backward(h, gain, dx, 1e-6, dx_residual=n)
                out += [dw]
            logits, nll, count, loss = h.clone(), torch.empty(M, device=cuda_device), torch.empty(1, dtype=torch.int32, device=cuda_device), torch.empty(2, device=cuda_device)
            _lib.check(lib.mcb_cross_entropy(logits.data_ptr(), targets.data_ptr(), nll.data_ptr(), count.data_ptr(), loss.data_ptr(), M, H, 1,
                                             B._dtype_code(logits), B._stream()))
            out += [h, grad_a, grad_b, logits, loss]
        return out

    try:
        _lib.check(lib.mcb_set_option(_lib.MCB_OPT_PDL, 0))
        want = chain()
        torch.cuda.synchronize()
    finally:
        _lib.check(lib.mcb_set_option(_lib.MCB_OPT_PDL, 1))
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(chain(), want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = chain()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(captured, want))
    assert _lib.device_status() == 0
