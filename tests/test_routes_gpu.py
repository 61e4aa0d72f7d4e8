"""GPU: which kernels a call launches.  The call is captured into a graph, whose nodes are
asked for their kernels' names: the tests that compare the forms with one another
compare what they say, and the rules of the dispatch hold on either side of their lines."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


class _KernelNode(ctypes.Structure):
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("smem", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p)]


def _kernels(rt, stream, call):
    """Names of the kernels that `call` launches on the stream; they do not run."""
    def ok(code):
        assert code == 0, code

    s, graph, count = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    ok(rt.cudaStreamBeginCapture(s, 1))
    try:
        call()
    finally:
        ok(rt.cudaStreamEndCapture(s, ctypes.byref(graph)))
    ok(rt.cudaGraphGetNodes(graph, None, ctypes.byref(count)))
    nodes = (ctypes.c_void_p * count.value)()
    ok(rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(count)))
    names = []
    for node in nodes:
        p, name = _KernelNode(), ctypes.c_char_p()
        ok(rt.cudaGraphKernelNodeGetParams(ctypes.c_void_p(node), ctypes.byref(p)))
        ok(rt.cudaFuncGetName(ctypes.byref(name), ctypes.c_void_p(p.func)))
        names.append(name.value.decode())
    ok(rt.cudaGraphDestroy(graph))
    return names


def _forms(names):
    return ["ring" if "pipe_kernel" in n else "barrier" if "fused_kernel" in n else "pass" for n in names]


def _smallest_ring_batch(logn, sms):
    """More tiles than resident CTAs and more than one transform (fft_fused2.cu)."""
    log_tile, ctas = (12, 2 * sms) if logn <= 16 else (13, sms)
    return max(2, ctas // (2 << (logn - log_tile)) + 1)


@pytest.fixture(scope="module")
def stream():
    torch = pytest.importorskip("torch")
    return torch.cuda.Stream()


@pytest.mark.parametrize("logn", range(15, 21))
def test_pairs(lib_built, stream, logn):
    import gbfft
    torch = pytest.importorskip("torch")
    n = 1 << logn
    least = _smallest_ring_batch(logn, torch.cuda.get_device_properties(0).multi_processor_count)
    x = torch.zeros((least * n + 1, 2), device="cuda")
    y = torch.zeros_like(x)
    with gbfft.Context(0) as ctx:
        def forms(a, b, batch):
            args = (a, b, n, batch, gbfft.FORWARD)
            ctx.c2c_device(*args, stream=stream.cuda_stream)  # makes the counters
            torch.cuda.synchronize()
            return _forms(_kernels(ctx._L, stream, lambda: ctx.c2c_device(*args, stream=stream.cuda_stream)))

        torch.cuda.synchronize()
        assert forms(x, y, least) == ["ring"]
        assert forms(x.data_ptr() + 8, y.data_ptr() + 8, least) == ["barrier"]
        assert forms(x, x, least) == ["pass", "pass"]
        # one transform less: the barrier form, or (radix 2^10 first) the ring with a CTA a tile
        if logn == 20:
            assert forms(x, y, 1) == ["barrier"]
        else:
            assert forms(x, y, least - 1) == ["ring" if logn == 19 else "barrier"]
        ctx.set_window(gbfft.WINDOW_HANN)
        assert forms(x, y, least) == ["barrier"]


@pytest.mark.parametrize("logn", range(21, 27))
def test_three_pass_sizes(lib_built, stream, logn):
    import gbfft
    torch = pytest.importorskip("torch")
    n = 1 << logn
    x = torch.zeros((n + 1, 2), device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    with gbfft.Context(0) as ctx:
        def forms(a, b):
            ctx.c2c_device(a, b, n, 1, gbfft.FORWARD, stream=stream.cuda_stream)
            torch.cuda.synchronize()
            return _forms(_kernels(ctx._L, stream, lambda: ctx.c2c_device(a, b, n, 1, gbfft.FORWARD,
                                                                          stream=stream.cuda_stream)))

        first = "ring" if logn == 26 else "pass"
        assert forms(x, y) == (["ring"] if logn <= 22 else [first, "ring"])
        assert forms(x, x) == [first, "ring"]
        assert forms(x.data_ptr() + 8, y.data_ptr() + 8) == ["pass", "barrier"]


def test_ragged(gpu_ctx, stream):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for count, offset, large in ((sms, 0, True), (2 * sms // 3, 0, False), (sms, 1, False)):
        # 2^16: eight tiles each; the ring from six tiles an SM on, at even offsets
        descs = [(offset + (k << 16), 16, -1) for k in range(count)]
        total = offset + (count << 16)
        x = torch.zeros((total + 1, 2), device="cuda")
        y = torch.zeros_like(x)
        plan = gpu_ctx.ragged_plan(descs)
        torch.cuda.synchronize()
        plan.execute(x, x, total, use_graph=False, stream=stream.cuda_stream)
        plan.wait(stream.cuda_stream)
        for a, b, ring in ((x.data_ptr(), y.data_ptr(), large), (x.data_ptr() + 8, y.data_ptr() + 8, False),
                           (x.data_ptr(), x.data_ptr(), False)):
            names = _kernels(gpu_ctx._L, stream, lambda: plan.execute(a, b, total, use_graph=False,
                                                                      stream=stream.cuda_stream))
            assert len(names) == 1 and ("fft_ragged_pipe_kernel" in names[0]) == ring, (count, offset, names)
            assert ring or "fft_ragged_kernel" in names[0], names
        plan.close()


@pytest.mark.parametrize("logn,prec,loop", [(8, 1, True), (12, 1, False), (12, 4, True), (13, 3, True), (13, 4, True), (14, 1, True),
                                            (14, 2, True), (14, 4, False)])
def test_split_single_pass_loop(lib_built, stream, logn, prec, loop):
    """A large launch takes the tile loop where that is the faster one (fft_rows_tc.cuh)."""
    import gbfft
    torch = pytest.importorskip("torch")
    n, batch = 1 << logn, (1 << 24) >> logn
    x = torch.zeros((n * batch, 2), device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    with gbfft.Context(0) as ctx:
        ctx.set_precision(prec)
        args = (x, y, n, batch, gbfft.FORWARD)
        ctx.c2c_device(*args, stream=stream.cuda_stream)
        torch.cuda.synchronize()
        names = _kernels(ctx._L, stream, lambda: ctx.c2c_device(*args, stream=stream.cuda_stream))
    assert len(names) == 1 and "fft_rows_tc_kernel" in names[0]
    assert ("Lb1E" in names[0]) == loop, names
