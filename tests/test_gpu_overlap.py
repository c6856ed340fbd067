"""GPU tests of tensor-core calls whose launches overlap the end of the kernel before them: a chain of steps in which every kernel reads
what the one before it wrote gives the bits of the same chain with the device idle between calls, on a stream, beside a copy and a
producer on other streams, and replayed from a graph."""
import pytest
import torch

import e_natten_b200 as na

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (kernel size, B, N, H, W, C, dtype): one tile; fewer tiles than SMs; several rounds; the largest size that overlaps in a graph, on a
# stream, and the first that does not
CASES = [(7, 1, 1, 7, 7, 32, torch.bfloat16), (13, 16, 4, 14, 14, 64, torch.float16), (9, 2, 3, 61, 50, 64, torch.bfloat16),
         (11, 2, 8, 40, 33, 128, torch.float16), (13, 3, 8, 28, 30, 128, torch.bfloat16), (7, 8, 4, 64, 64, 32, torch.float16),
         (9, 16, 4, 64, 64, 64, torch.bfloat16), (7, 1, 3, 257, 341, 32, torch.bfloat16)]


def _chain(x, ks, between):
    """Three steps; the gradients of one, normalised, are the inputs of the next."""
    outs = []
    q, k, v, d_o = x
    for _ in range(3):
        between()
        o, lse = na.natten2d_forward(q, k, v, ks, scale=q.shape[-1] ** -0.5)
        between()
        d_q, d_k, d_v = na.natten2d_backward(q, k, v, o, lse, d_o, ks, scale=q.shape[-1] ** -0.5)
        between()
        outs += [o, lse, d_q, d_k, d_v]
        q, k, v, d_o = d_k, d_q, o, d_v
    # and forwards that read the forward before them, with nothing in between
    for _ in range(3):
        between()
        o, lse = na.natten2d_forward(o, k, v, ks, scale=1.0)
        outs += [o, lse]
    return outs


def _inputs(B, N, H, W, C, dtype):
    g = torch.Generator().manual_seed(H * W + C)
    return [torch.randn(B, N, H, W, C, generator=g).to(DEV, dtype) for _ in range(4)]


def _same(got, want):
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), f"result {i}"


@pytest.mark.parametrize("ks,B,N,H,W,C,dtype", CASES)
def test_chain_on_a_stream(ks, B, N, H, W, C, dtype):
    x = _inputs(B, N, H, W, C, dtype)
    want = _chain(x, ks, torch.cuda.synchronize)
    for _ in range(3):
        _same(_chain(x, ks, lambda: None), want)


@pytest.mark.parametrize("ks,B,N,H,W,C,dtype", CASES[1:6])
def test_chain_replayed(ks, B, N, H, W, C, dtype):
    x = _inputs(B, N, H, W, C, dtype)
    want = _chain(x, ks, torch.cuda.synchronize)
    side = torch.cuda.Stream()
    held = [torch.zeros_like(t) for t in x]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        # the inputs come from a branch of their own, which joins before the first launch
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for h, t in zip(held, x):
                h.copy_(t)
        torch.cuda.current_stream().wait_stream(side)
        got = _chain(held, ks, lambda: None)
    for _ in range(3):
        for h in held:
            h.zero_()
        graph.replay()
        _same(got, want)


@pytest.mark.parametrize("ks,B,N,H,W,C,dtype", CASES[1:4])
def test_inputs_from_another_stream(ks, B, N, H, W, C, dtype):
    x = _inputs(B, N, H, W, C, dtype)
    want = na.natten2d_forward(*x[:3], ks, scale=1.0)
    other = [t.flip(0).contiguous() for t in x[:3]]
    pinned = x[0].cpu().pin_memory()
    held = [torch.zeros_like(t) for t in x[:3]]
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(main):
            first = na.natten2d_forward(*other, ks, scale=1.0)     # a kernel of ours right before the wait
        with torch.cuda.stream(side):
            side.wait_stream(main)
            for h, t in zip(held[1:], x[1:3]):
                h.copy_(t)
        with torch.cuda.stream(main):
            main.wait_stream(side)
            held[0].copy_(pinned, non_blocking=True)
            got = na.natten2d_forward(*held, ks, scale=1.0)
            for h in held:
                h.zero_()
        torch.cuda.synchronize()
        _same(got, want)
        del first
