"""GPU: an error of the caller's that is still pending stays so over a call that succeeds."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn,batch", [(10, 9), (16, 40)])
@pytest.mark.parametrize("captured", [False, True])
def test_pending_error_is_left_alone(lib_built, logn, batch, captured):
    import gbfft
    torch = pytest.importorskip("torch")
    n = 1 << logn
    x = torch.view_as_complex(torch.randn(batch, n, 2, device="cuda"))
    y = torch.empty_like(x)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with gbfft.Context(0) as ctx:
        ctx.c2c_device(x, y, n, batch, gbfft.FORWARD, stream=stream.cuda_stream)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            if captured:
                graph.capture_begin()
            code = ctx._L.cudaSetDevice(1 << 20)
            ctx.c2c_device(x, y, n, batch, gbfft.FORWARD, stream=stream.cuda_stream)
            pending = ctx._L.cudaGetLastError()
            if captured:
                graph.capture_end()
        assert code != 0 and pending == code
