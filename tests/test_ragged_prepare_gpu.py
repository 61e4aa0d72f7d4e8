"""GPU: what a ragged plan keeps between calls -- tables and queues -- is complete or not
there: after a first call under capture, and whichever of the two forms (ring of tiles,
barrier) the calls before took.  A time-out stays reported until it is read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_REL_L2 = 2e-6


def _descs(sizes, seed=5):
    """Transforms of these log2 sizes back to back, directions mixed, at even offsets."""
    rng = np.random.default_rng(seed)
    descs, off = [], 2
    for L in sizes:
        descs.append((off, int(L), int(rng.choice([-1, 1]))))
        off += max(2, 1 << int(L))
    return descs, off


def _large(seed=5):
    """Enough two-pass transforms of 2^14 .. 2^18 for the ring (fft_ragged.cu, rag_pipe_pays)."""
    rng = np.random.default_rng(seed)
    return _descs(list(rng.permutation(list(range(8, 19)) + [int(v) for v in rng.choice(range(14, 19), 130)])), seed)


def _small():
    return _descs(list(range(19)))


def _data(torch, total):
    x = torch.view_as_complex(torch.randn(total, 2, generator=torch.Generator("cuda").manual_seed(total), device="cuda"))
    return x, torch.full_like(x, float("nan"))


def _check(torch, x, y, descs):
    for off, L, d in descs:
        a = x[off:off + (1 << L)].to(torch.complex128)
        want = torch.fft.fft(a) if d < 0 else torch.fft.ifft(a)
        err = (torch.linalg.vector_norm(y[off:off + (1 << L)] - want) / torch.linalg.vector_norm(want)).item()
        assert err <= TOL_REL_L2, (off, L, d, err)


@pytest.mark.parametrize("prec,large", [(0, False), (0, True), (1, False)])
def test_tables_after_a_first_call_under_capture(lib_built, prec, large):
    """A plan's first call makes its tables and cannot be captured; it is refused, and the
    next ordinary call makes them."""
    import gbfft
    torch = pytest.importorskip("torch")
    descs, total = _large() if large else _small()
    x, y = _data(torch, total)
    with gbfft.Context(0) as ctx:
        ctx.set_precision(prec)
        plan = ctx.ragged_plan(descs)
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="relaxed")
            try:
                with pytest.raises(gbfft.GbfftError):
                    plan.execute(x, y, total, use_graph=False, stream=stream.cuda_stream)
            finally:
                try:
                    graph.capture_end()
                except RuntimeError:
                    ctx._L.cudaGetLastError()
        ctx._L.cudaGetLastError()
        for graphed in (False, True):
            y.fill_(float("nan"))
            torch.cuda.synchronize()
            plan.execute(x, y, total, use_graph=graphed)
            plan.wait()
            _check(torch, x, y, descs)
        plan.close()


@pytest.mark.parametrize("first,then", [(0, 8), (8, 0)])
def test_one_ordinary_call_prepares_both_forms(gpu_ctx, first, then):
    """A call on 16-byte boundaries takes the ring, one 8 bytes on the barrier form; either
    makes ready what the other needs under capture."""
    torch = pytest.importorskip("torch")
    descs, total = _large()
    x, y = _data(torch, total + 1)
    xa, ya = x[1:].clone(), torch.full_like(x[1:], float("nan"))
    buf = {0: (xa.data_ptr(), ya.data_ptr()), 8: (x.data_ptr() + 8, y.data_ptr() + 8)}
    plan = gpu_ctx.ragged_plan(descs)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    plan.execute(*buf[first], total, use_graph=False, stream=stream.cuda_stream)
    plan.wait(stream.cuda_stream)
    with torch.cuda.graph(graph, stream=stream):
        plan.execute(*buf[then], total, use_graph=False, stream=stream.cuda_stream)
    for _ in range(2):
        y.fill_(float("nan"))
        ya.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        _check(torch, xa, ya if then == 0 else y[1:], descs)
    plan.close()


@pytest.mark.parametrize("large", [False, True])
def test_a_time_out_is_reported_by_the_next_wait(gpu_ctx, large):
    """A run that gave up, then a good one with no wait between: the wait reports the first."""
    import gbfft
    torch = pytest.importorskip("torch")
    descs, total = _large() if large else _small()
    x, y = _data(torch, total)
    plan = gpu_ctx.ragged_plan(descs)
    plan.set(gbfft.RAGGED_OPT_SPIN_LIMIT, 2000)
    plan.set(gbfft.RAGGED_OPT_TEST_DROP_PRODUCERS, 1)
    plan.execute(x, y, total, use_graph=False)
    plan.set(gbfft.RAGGED_OPT_TEST_DROP_PRODUCERS, 0)
    plan.set(gbfft.RAGGED_OPT_SPIN_LIMIT, 1 << 22)
    plan.execute(x, y, total, use_graph=False)
    with pytest.raises(gbfft.GbfftError) as e:
        plan.wait()
    assert e.value.status == gbfft.ERR_TIMEOUT
    _check(torch, x, y, descs)
    plan.execute(x, y, total, use_graph=True)
    plan.wait()  # reported once
    plan.close()
