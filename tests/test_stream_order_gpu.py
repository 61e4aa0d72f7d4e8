"""GPU: launches that follow one another in a stream without a wait between them.

Each kernel may be brought up while the one before it runs; what it reads and writes
must still be ordered.  A chain of in-place and out-of-place transforms of one buffer
set, enqueued back to back, gives the same bits as the same chain with the device
idle between calls; so does the chain with other kernels, copies and memory sets
between the calls, and the chain replayed from a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(0, 7, 0), (3, 1, 0), (6, 33, 0), (10, 9, 0), (12, 64, 0), (13, 40, 0), (14, 9, 0),  # one pass
          (15, 3, 0), (16, 40, 0), (18, 2, 0), (20, 1, 0), (20, 3, 0),  # pass pairs, both forms
          (21, 1, 0), (22, 2, 0), (23, 1, 0), (26, 1, 0),  # two and three passes
          (8, 40, 1), (11, 5000, 1), (16, 8, 1), (9, 33, 3), (13, 20, 4)]  # split forms


def _chain(ctx, gbfft, torch, x, n, batch, stream, between):
    y, z = torch.empty_like(x), torch.empty_like(x)
    outs = []
    for k in range(6):
        ctx.c2c_device(x, y, n, batch, gbfft.FORWARD, stream=stream)
        between(k)
        ctx.c2c_device(y, y, n, batch, gbfft.INVERSE, stream=stream)
        ctx.c2c_device(y, z, n, batch, gbfft.FORWARD, stream=stream)
        between(k)
        ctx.c2c_device(z, x, n, batch, gbfft.INVERSE, stream=stream)
    outs += [x, y, z]
    return outs


@pytest.mark.parametrize("logn,batch,prec", SHAPES)
def test_back_to_back_launches(lib_built, logn, batch, prec):
    import gbfft
    torch = pytest.importorskip("torch")
    n = 1 << logn
    g = torch.Generator(device="cuda")
    g.manual_seed(900 + logn)
    x0 = torch.view_as_complex(torch.randn(batch * n, 2, generator=g, device="cuda"))
    side = torch.zeros(1 << 16, device="cuda")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()  # one stream throughout: a context's counters are a stream's own
    st = stream.cuda_stream
    with gbfft.Context(0) as ctx, torch.cuda.stream(stream):
        ctx.set_precision(prec)
        want = _chain(ctx, gbfft, torch, x0.clone(), n, batch, st, lambda k: torch.cuda.synchronize())
        torch.cuda.synchronize()

        def others(k):
            side.add_(1.0)
            if k % 2:
                side.zero_()
                side[1:].copy_(side[:-1].clone())

        for between in (lambda k: None, others):
            got = _chain(ctx, gbfft, torch, x0.clone(), n, batch, st, between)
            torch.cuda.synchronize()
            for a, b in zip(got, want):
                assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))
        # from a graph (the calls above have made the workspaces)
        x = x0.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = _chain(ctx, gbfft, torch, x, n, batch, st, lambda k: None)
        x.copy_(x0)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))
