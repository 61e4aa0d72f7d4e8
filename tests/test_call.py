"""The extension module's c2c (gbfft/_call.c) on the CPU: what it passes on, and what it
leaves to the ctypes path by answering None.  The library function is a stand-in."""
import ctypes
import importlib.machinery
import importlib.util
import os

import numpy as np
import pytest


class _Tensor:
    def __init__(self, p):
        self.p = p

    def data_ptr(self):
        return self.p


class _Broken:
    def data_ptr(self):
        raise ValueError("no storage")


@pytest.fixture(scope="module")
def c2c():
    import sys
    import gbfft
    b = sys.modules[gbfft.build.__module__]
    os.makedirs(b.LIB_DIR, exist_ok=True)
    b._build_call(False)
    if not os.path.exists(b.CALL_PATH):
        pytest.skip("no Python headers or C compiler")
    loader = importlib.machinery.ExtensionFileLoader("_gbfft_call", b.CALL_PATH)
    m = importlib.util.module_from_spec(importlib.util.spec_from_loader("_gbfft_call", loader))
    loader.exec_module(m)
    return m.c2c


def test_arguments_and_what_is_left_to_ctypes(c2c):
    seen = []
    u64, vp, i = ctypes.c_uint64, ctypes.c_void_p, ctypes.c_int
    fn = ctypes.CFUNCTYPE(i, vp, vp, vp, u64, u64, i, vp)(lambda *a: seen.append(a) or 7)
    f = ctypes.cast(fn, vp).value
    big = (1 << 63) + 16
    assert c2c(f, 5, _Tensor(big), 48, 1024, 9, -1, None) == 7
    assert c2c(f, 5, 0, _Tensor(64), 1 << 40, 0, 1, 77) == 7
    assert seen == [(5, big, 48, 1024, 9, -1, None), (5, None, 64, 1 << 40, 0, 1, 77)]
    ok = [f, 5, 16, 48, 1024, 9, -1, None]
    for pos, bad in ((2, None), (2, 1.5), (2, np.zeros(4, np.complex64)), (3, _Broken()), (3, -1), (4, -1), (4, 1 << 64),
                     (4, np.int64(8)), (4, 8.0), (5, True), (5, None), (6, 1 << 40), (6, 1.0), (7, "0"), (7, np.int64(0)),
                     (7, -1), (0, 0)):
        args = list(ok)
        args[pos] = bad
        assert c2c(*args) is None, (pos, bad)
    assert c2c(*ok[:7]) is None
    assert len(seen) == 2


@pytest.mark.gpu
def test_same_results_and_errors_as_ctypes(lib_built):
    import gbfft
    torch = pytest.importorskip("torch")
    x = torch.view_as_complex(torch.randn(9, 1024, 2, device="cuda"))
    outs = []
    with gbfft.Context(0) as ctx:
        for direct in (True, False):
            if not direct:
                ctx._c2c = None
            y = torch.zeros_like(x)
            ctx.c2c_device(x, y, 1024, 9, gbfft.FORWARD, stream=torch.cuda.current_stream().cuda_stream)
            ctx.c2c_device(y.data_ptr(), y.data_ptr(), np.uint64(1024).item(), 9)
            torch.cuda.synchronize()
            outs.append(y)
            for args, status in (((x, y, 1000, 9), gbfft.ERR_INVALID_SIZE), ((x, y, 1024, 9, 3), gbfft.ERR_INVALID_ARGUMENT),
                                 ((0, y, 1024, 9), gbfft.ERR_INVALID_ARGUMENT)):
                with pytest.raises(gbfft.GbfftError) as e:
                    ctx.c2c_device(*args)
                assert e.value.status == status
            with pytest.raises(TypeError):
                ctx.c2c_device(None, y, 1024, 9)
            with pytest.raises(ctypes.ArgumentError):
                ctx.c2c_device(x, y, 1024.0, 9)
    assert torch.equal(torch.view_as_real(outs[0]), torch.view_as_real(outs[1]))
    with pytest.raises(gbfft.GbfftError):
        ctx.c2c_device(x, y, 1024, 9)  # closed
