"""GPU: the warp-column pass pairs (fft_pipe.cuh) against the barrier form of the
same pairs and against FP64.

Buffers on 16-byte boundaries take the warp-column form once a launch has more
tiles than resident CTAs; the same rows at an odd multiple of 8 bytes take the
barrier form.  Both do the same arithmetic: the same bits, except at 2^21 and
2^22, which take two passes instead of three (FP64 bound only).  Batches: the
smallest that take the form, odd ones, one with several rounds of the ring."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_REL_L2 = 2e-6


@pytest.mark.parametrize("logn,batch", [(15, 20), (15, 301), (16, 11), (16, 203), (17, 5), (17, 67), (18, 3), (18, 33),
                                        (19, 1), (19, 2), (19, 13), (20, 2), (20, 5), (21, 1), (21, 3), (22, 1), (22, 3), (23, 1),
                                        (24, 1), (25, 1), (26, 1), (26, 2)])
def test_pipe_matches_barrier_form_and_fp64(lib_built, logn, batch):
    import gbfft
    torch = pytest.importorskip("torch")
    n = 1 << logn
    g = torch.Generator(device="cuda")
    g.manual_seed(700 + logn)
    x = torch.view_as_complex(torch.randn(batch * n + 1, 2, generator=g, device="cuda"))
    a = x[1:].clone()  # 16-byte aligned copy of the rows at x + 8 bytes
    assert a.data_ptr() % 16 == 0 and x.data_ptr() % 16 == 0
    with gbfft.Context(0) as ctx:
        for direction in (gbfft.FORWARD, gbfft.INVERSE):
            y = torch.full_like(a, float("nan"))
            z = torch.full_like(x, float("nan"))
            for _ in range(2):  # the second launch finds the counters cleared
                ctx.c2c_device(a, y, n, batch, direction, stream=torch.cuda.current_stream().cuda_stream)
            ctx.c2c_device(x.data_ptr() + 8, z.data_ptr() + 8, n, batch, direction,
                           stream=torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            if logn not in (21, 22):
                assert torch.equal(torch.view_as_real(y), torch.view_as_real(z[1:]))
            assert torch.isnan(z[0].real)
            for row in {0, batch // 2, batch - 1}:
                r = a[row * n:(row + 1) * n].to(torch.complex128)
                want = torch.fft.fft(r) if direction == gbfft.FORWARD else torch.fft.ifft(r)
                got = y[row * n:(row + 1) * n].to(torch.complex128)
                assert ((got - want).norm() / want.norm()).item() <= TOL_REL_L2
        ctx.c2c_host(np.zeros((1, 1 << 15), np.complex64))  # reports a device wait that gave up, if any did


def test_two_pass_launch_of_2_21_and_2_22(lib_built):
    """One launch out of place; in place and with a window the three-pass plan."""
    import gbfft
    torch = pytest.importorskip("torch")
    for logn in (21, 22):
        n = 1 << logn
        x = torch.view_as_complex(torch.randn(2, n, 2, device="cuda"))
        with gbfft.Context(0) as ctx:
            for in_place, window, launches in ((False, False, 1), (True, False, 2), (False, True, 2)):
                ctx.set_window(gbfft.WINDOW_HANN if window else gbfft.WINDOW_NONE)
                a = x.clone()
                y = a if in_place else torch.empty_like(a)
                before = ctx.launch_count()
                ctx.c2c_device(a, y, n, 2, gbfft.FORWARD, stream=torch.cuda.current_stream().cuda_stream)
                torch.cuda.synchronize()
                assert ctx.launch_count() - before == launches
                r = x.to(torch.complex128)
                if window:
                    i = torch.arange(n, dtype=torch.float64, device="cuda")
                    r = r * (0.5 * (1 - torch.cos(2 * torch.pi * i / (n - 1))))
                want = torch.fft.fft(r)
                assert ((y.to(torch.complex128) - want).norm() / want.norm()).item() <= TOL_REL_L2


def test_pipe_under_capture_and_on_two_streams(lib_built):
    import gbfft
    torch = pytest.importorskip("torch")
    n, batch = 1 << 16, 64
    xs = [torch.view_as_complex(torch.randn(batch, n, 2, device="cuda")) for _ in range(2)]
    ys = [torch.empty_like(x) for x in xs]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    with gbfft.Context(0) as ctx:
        for _ in range(4):
            for x, y, s in zip(xs, ys, streams):
                ctx.c2c_device(x, y, n, batch, gbfft.FORWARD, stream=s.cuda_stream)
        torch.cuda.synchronize()
        want = [y.clone() for y in ys]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            ctx.c2c_device(xs[0], ys[0], n, batch, gbfft.FORWARD, stream=streams[0].cuda_stream)
        for _ in range(3):
            ys[0].zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(torch.view_as_real(ys[0]), torch.view_as_real(want[0]))
    for x, y in zip(xs, want):
        ref = torch.fft.fft(x[:2].to(torch.complex128))
        assert ((y[:2].to(torch.complex128) - ref).norm() / ref.norm()).item() <= TOL_REL_L2
