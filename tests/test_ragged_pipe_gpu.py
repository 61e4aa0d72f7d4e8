"""GPU: ragged batches large enough for the warp-column kernel (fft_ragged_pipe.cu),
against FP64 per transform, and the same plan on buffers that take the barrier form
(in place; 8 bytes off a 16-byte boundary).

The set has every size 2^0 .. 2^18 in both directions; `gap` samples between
transforms put offsets at every even residue of a tile row (an odd gap keeps the whole
plan on the barrier form)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_REL_L2 = 2e-6


def _set(seed, gap, big, count):
    """All sizes in both directions, then `count` transforms of the sizes `big`."""
    rng = np.random.default_rng(seed)
    sizes = list(range(0, 19)) * 2 + [int(v) for v in rng.choice(big, size=count)]
    dirs = [-1] * 19 + [1] * 19 + [int(v) for v in rng.choice([-1, 1], size=count)]
    descs, off = [], 2
    for k in rng.permutation(len(sizes)):
        descs.append((off, sizes[k], dirs[k]))
        off += (1 << sizes[k]) + (1 if sizes[k] == 0 and gap % 2 == 0 else 0) + gap  # the next offset: even
    return descs, off


def _check(torch, x, y, descs):
    for off, L, d in descs:
        a = x[off:off + (1 << L)].to(torch.complex128)
        want = torch.fft.fft(a) if d < 0 else torch.fft.ifft(a)
        err = (torch.linalg.vector_norm(y[off:off + (1 << L)] - want) / torch.linalg.vector_norm(want)).item()
        assert err <= TOL_REL_L2, (off, L, d, err)


@pytest.mark.parametrize("seed,gap,big,count", [(1, 0, (14,), 640), (2, 2, (15,), 330), (3, 6, (16,), 170), (4, 14, (17,), 90),
                                                (5, 0, (18,), 48), (6, 10, (14, 15, 16, 17, 18), 130),
                                                (7, 3, (14, 15, 16, 17, 18), 130)])
def test_large_ragged_sets(gpu_ctx, seed, gap, big, count):
    torch = pytest.importorskip("torch")
    descs, total = _set(seed, gap, big, count)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.view_as_complex(torch.randn(total, 2, generator=g, device="cuda"))
    y = torch.full_like(x, float("nan"))
    plan = gpu_ctx.ragged_plan(descs)
    for graph in (False, True, True):
        plan.execute(x, y, total, use_graph=graph)
        plan.wait()
    _check(torch, x, y, descs)
    outside = torch.ones(total, dtype=torch.bool, device="cuda")
    for off, L, _ in descs:
        outside[off:off + (1 << L)] = False
    assert torch.isnan(y[outside].real).all()  # as full_like left them: NaN + 0i
    # the same plan 8 bytes on, and in place
    xo = torch.cat([x[:1], x])
    yo = torch.full_like(xo, float("nan"))
    plan.execute(xo.data_ptr() + 8, yo.data_ptr() + 8, total, use_graph=False)
    plan.wait()
    _check(torch, x, yo[1:], descs)
    z = x.clone()
    plan.execute(z, z, total, use_graph=False)
    plan.wait()
    _check(torch, x, z, descs)
    plan.close()


def test_large_ragged_set_dependency_wait_times_out(gpu_ctx):
    """The first-pass items are dropped on the host: the loaders' bounded waits give up,
    the host reports the time-out and the plan runs again afterwards."""
    import gbfft
    torch = pytest.importorskip("torch")
    descs, total = _set(8, 2, (16, 17, 18), 90)
    x = torch.view_as_complex(torch.randn(total, 2, device="cuda"))
    y = torch.zeros_like(x)
    plan = gpu_ctx.ragged_plan(descs)
    plan.set(gbfft.RAGGED_OPT_SPIN_LIMIT, 2000)
    plan.set(gbfft.RAGGED_OPT_TEST_DROP_PRODUCERS, 1)
    plan.execute(x, y, total, use_graph=False)
    with pytest.raises(gbfft.GbfftError) as e:
        plan.wait()
    assert e.value.status == gbfft.ERR_TIMEOUT
    plan.set(gbfft.RAGGED_OPT_TEST_DROP_PRODUCERS, 0)
    plan.set(gbfft.RAGGED_OPT_SPIN_LIMIT, 1 << 20)
    plan.execute(x, y, total, use_graph=True)
    plan.wait()
    _check(torch, x, y, descs)
    plan.close()
