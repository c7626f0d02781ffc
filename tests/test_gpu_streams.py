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
