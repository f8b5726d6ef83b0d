"""Calls that overlap: two streams, two threads on one stream, a captured call whose scratch was outgrown since, and a kernel
that is set up while the one ahead of it still writes what it reads."""

import threading

import pytest
import torch

import algebraic_transformer_b200 as A
from algebraic_transformer_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def randn(shape, seed, dtype=torch.bfloat16):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(DEV)


def decode_inputs(seed, B=2, H=6, Tk=5000, D=64):
    return tuple(randn((B, H, n, D), seed + i) for i, n in enumerate((1, Tk, Tk)))


def train_inputs(seed, B=1, H=4, T=700, D=64):
    q, k, v, d_o = (randn((B, H, T, D), seed + i) for i in range(4))
    sink = torch.zeros(H, device=DEV)
    o, stat, which = A.flash_attention(q, k, v, sink, kind="asinh", n=16, c=8.0, block=T, range_guard=True, return_stat=True)
    return q, k, v, o, d_o, stat, which, sink


def decode(t):
    return [A.decode_attention(*t, n=16, c=8.0)]


def backward(t):
    return list(A.flash_attention_backward(*t, n=16, c=8.0))[:3]       # dsink is a sum by atomics, in any order


def forward(t):
    return [A.flash_attention(*t[:3], t[7], kind="asinh", n=16, c=8.0, block=t[0].shape[2], range_guard=True)]


@pytest.mark.parametrize("call,make", [(decode, decode_inputs), (backward, train_inputs), (forward, train_inputs)])
def test_two_streams_and_two_threads(call, make):
    cases = [make(10), make(20)]
    want = [call(c) for c in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(call(cases[i]))
    torch.cuda.synchronize()
    shared = torch.cuda.Stream()

    def work(i):
        with torch.cuda.stream(shared):
            for _ in range(20):
                got[i].append(call(cases[i]))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(2):
        assert len(got[i]) == 40
        for out in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(out, want[i]))


@pytest.mark.parametrize("call,make,small,large", [(decode, decode_inputs, dict(Tk=900), dict(B=16, Tk=900)),
                                                   (backward, train_inputs, dict(T=300), dict(T=900, B=8))])
def test_captured_call_outlives_larger_ones(call, make, small, large):
    a, b = make(30, **small), make(40, **large)
    want = call(a)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        call(a)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        out = call(a)
    for _ in range(3):
        call(b)
        filler = [torch.full((n,), 255, dtype=torch.uint8, device=DEV) for n in (1 << 10, 1 << 14, 1 << 18, 1 << 21)]
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(out, want))
        assert all(bool((f == 255).all()) for f in filler)


def test_gains_written_by_the_kernel_ahead():
    """The projection kernel moves in before the kernel ahead has finished; every input has to wait for that one, gains too."""
    M, K, H, D = 256, 128, 2, 64
    x, w = randn((M, K), 50), randn((3 * H * D, K), 51)
    cos, sin = A.cayley_table_geometric(D, M, device=DEV)
    gains = torch.rand((40, D), generator=torch.Generator().manual_seed(52)).add_(0.5).to(DEV)
    gain = torch.empty(D, device=DEV)

    def project(g):
        return ops.qkv_projection(x, w, H, M, cos.bfloat16(), sin.bfloat16(), g, g)
    want = [project(g) for g in gains]
    torch.cuda.synchronize()
    got = []
    for g in gains:
        gain.copy_(g)
        got.append(project(gain))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
