"""GPU: 2^21 and 2^22, which take one two-pass launch where the buffers allow it, in the
calls that cannot: under capture after an ordinary call that could, and with an output
that overlaps the input."""
import pytest

pytestmark = pytest.mark.gpu

TOL_REL_L2 = 2e-6


def _rel(torch, got, want):
    return (torch.linalg.vector_norm(got.to(torch.complex128) - want) / torch.linalg.vector_norm(want)).item()


@pytest.mark.parametrize("logn", [21, 22])
@pytest.mark.parametrize("form", ["in place", "8 bytes on", "noise"])
def test_capture_after_one_ordinary_call(lib_built, logn, form):
    """One ordinary call of a size on a stream makes ready what any call of that size and
    batch on it needs."""
    import gbfft
    torch = pytest.importorskip("torch")
    n, batch = 1 << logn, 3
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    buf = torch.view_as_complex(torch.randn(batch * n + 1, 2, device="cuda"))
    out = torch.full_like(buf, float("nan"))
    x = buf[1:].clone()
    y = torch.empty_like(x)
    want = torch.fft.fft(x.view(batch, n).to(torch.complex128)).view(-1)
    torch.cuda.synchronize()
    with gbfft.Context(0) as ctx:
        st = stream.cuda_stream
        ctx.c2c_device(x, y, n, batch, gbfft.FORWARD, stream=st)
        stream.synchronize()
        a = x.clone()
        if form == "noise":
            with gbfft.Context(0) as other:
                other.set_noise(7, 0.1)
                other.c2c_device(x, y, n, batch, gbfft.FORWARD, stream=st)
                stream.synchronize()
            want, y = y, torch.empty_like(x)
            ctx.set_noise(7, 0.1)
        args = {"in place": (a, a), "8 bytes on": (buf.data_ptr() + 8, out.data_ptr() + 8), "noise": (x, y)}[form]
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            ctx.c2c_device(*args, n, batch, gbfft.FORWARD, stream=st)
        a.copy_(x)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = {"in place": a, "8 bytes on": out[1:], "noise": y}[form]
        assert _rel(torch, got, want.to(torch.complex128)) <= TOL_REL_L2


@pytest.mark.parametrize("logn", [21, 22])
@pytest.mark.parametrize("shift", [2, 4096, -4096, (1 << 21) + 2, -(1 << 21) - 2])
def test_output_that_overlaps_the_input(lib_built, logn, shift):
    """Samples apart by `shift`: the three-pass form reads all of the input before it writes
    any of the output."""
    import gbfft
    torch = pytest.importorskip("torch")
    n, batch = 1 << logn, 3
    buf = torch.view_as_complex(torch.randn(batch * n + abs(shift), 2, device="cuda"))
    i, o = (0, shift) if shift > 0 else (-shift, 0)
    x, y = buf[i:i + batch * n], buf[o:o + batch * n]
    want = torch.fft.ifft(x.view(batch, n).to(torch.complex128)).view(-1)
    with gbfft.Context(0) as ctx:
        ctx.c2c_device(x, y, n, batch, gbfft.INVERSE, stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    assert _rel(torch, y, want) <= TOL_REL_L2
