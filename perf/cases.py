"""The transforms that a program asks of this library, as cases to be timed.

A case is one call pattern through the public entry points: device-resident
batches (`Context.c2c_device`), the same with the tensor-core split precisions
or a Hann window, ragged batches (`Context.ragged_plan`), and host rows through
the reference-style executor (`GpuFft.fft` / `ifft`).  The sizes are those of
the benchmark configurations, the size sweep (N = 2^5 .. 2^26) and the rivalry
leaderboard, with odd batches beside the round ones.

Fields of a case: kind (device | ragged | rows), logn, batch, op (fwd | inv |
both: forward, then inverse of the result), inplace, prec (0 FP32, 1 FP16 hi+lo,
2 BF16x3, 3 TF32, 4 BF16x6), hann, data (normal | uniform | tones).
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(1, os.path.join(_ROOT, "wgls-rs-fft_gb300"))

import gbfft  # noqa: E402

TC_KINDS = (1, 2, 3, 4)


def _case(kind, logn, batch, op="fwd", inplace=False, prec=0, hann=False, data="normal", **more):
    return dict(kind=kind, logn=logn, batch=batch, op=op, inplace=inplace, prec=prec, hann=hann, data=data, **more)


def listed():
    return [
        # the reference's own small configuration (8 rows and one more of N = 1024), forward and back:
        # a caller that transforms a handful of rows at a time pays for the calls and launches
        dict(_case("device", 10, 9, "both", data="uniform"), name="small_n1024_b9_both"),
        # the drop-in call of a reference user: 64 separate host rows in, 64 new ones out
        # (the rivalry leaderboard's N = 65536 entry)
        dict(_case("rows", 16, 64), name="host_rows_n65536_b64"),
        # many short spectra, a batch that is no multiple of a tile
        dict(_case("device", 9, 100003, "inv"), name="n512_b100003_inv"),
        # the headline configuration: 512 MB of N = 4096 rows
        dict(_case("device", 12, 16384), name="n4096_b16384_fwd"),
        # windowed analysis of longer rows: Hann applied as the samples are loaded
        dict(_case("device", 13, 8192, hann=True), name="n8192_b8192_hann"),
        # the size sweep's longest row that one block holds, back from the spectrum
        dict(_case("device", 14, 4096, "inv"), name="n16384_b4096_inv"),
        # mid-size spectra, the size the precision forms are compared at
        dict(_case("device", 16, 1024), name="n65536_b1024_fwd"),
        # long rows, an odd batch, inverse
        dict(_case("device", 19, 101, "inv"), name="n524288_b101_inv"),
        # large-N configuration: 4M-point rows
        dict(_case("device", 22, 16), name="n4194304_b16_fwd"),
        # one 64M-point transform, back from the spectrum
        dict(_case("device", 26, 1, "inv"), name="n67108864_b1_inv"),
        # the split-precision form on the tensor cores: tones over 120 dB
        dict(_case("device", 16, 1024, prec=1, data="tones"), name="tc_fp16_n65536_b1024"),
        # a ragged batch: sizes 2^8 .. 2^18 and directions mixed, one launch
        dict(_case("ragged", 18, 1250, "both", data="uniform"), name="ragged_1250"),
    ]


def draw(rng: random.Random):
    kind = rng.choices(("device", "split", "ragged", "rows"), (60, 20, 10, 10))[0]
    if kind == "ragged":
        return _case("ragged", rng.randint(12, 18), int(2 ** rng.uniform(4, 10.2)), "both", data="uniform",
                     prec=rng.choice((0, 0, 1)))
    if kind == "rows":
        total, logn = rng.uniform(10, 22), rng.randint(8, 18)
        batch = min(60, max(1, int(2 ** (total - logn))))
        return _case("rows", logn, batch, rng.choice(("fwd", "inv")))
    total = rng.uniform(14, 25.9)
    if kind == "split":
        logn = rng.randint(8, 18)
        prec = rng.choice(TC_KINDS)
        if prec == 3 and logn == 14:
            logn = 13  # TF32 has no single-pass form of 2^14
        return _case("device", logn, max(1, int(2 ** (total - logn))), rng.choice(("fwd", "inv")), prec=prec,
                     data="tones")
    logn = rng.randint(5, 24)
    batch = max(1, int(2 ** (total - logn)))
    op = rng.choice(("fwd", "inv", "both"))
    return _case("device", logn, batch, op, inplace=op == "both" and rng.random() < 0.5, hann=rng.random() < 0.15,
                 data=rng.choice(("normal", "uniform")))


# ---- inputs ----------------------------------------------------------------

def _input(case, seed, rows, n, device):
    """[rows, n] complex64 made from the seed on the device."""
    g = torch.Generator(device=device)
    g.manual_seed(seed * 7919 + case["logn"])
    if case["data"] == "uniform":
        return torch.view_as_complex(torch.rand(rows, n, 2, generator=g, device=device) * 2 - 1)
    x = torch.view_as_complex(torch.randn(rows, n, 2, generator=g, device=device))
    if case["data"] == "tones":
        # 64 tones a row, amplitudes log-uniform in [1e-3, 1e3], over noise of 1e-2
        k = 64
        spec = torch.zeros(rows, n, dtype=torch.complex64, device=device)
        bins = torch.randint(0, n // k, (rows, k), generator=g, device=device)
        bins += torch.arange(k, device=device) * (n // k)  # one in each 64th of the band: all different
        amp = 10.0 ** (6.0 * torch.rand(rows, k, generator=g, device=device) - 3.0)
        ph = 2.0 * math.pi * torch.rand(rows, k, generator=g, device=device)
        spec.scatter_(1, bins, torch.polar(amp * n, ph))
        x = torch.fft.ifft(spec, dim=1) + 1e-2 * x
    return x


def _ragged_set(case):
    """log2 N uniform on 8 .. logn, directions 50/50, packed back to back: the
    plan that a program keeps for its mix of rows."""
    r = np.random.RandomState(case["batch"])
    logs = r.randint(8, case["logn"] + 1, case["batch"])
    dirs = np.where(r.rand(case["batch"]) < 0.5, gbfft.FORWARD, gbfft.INVERSE)
    sizes = np.left_shift(np.int64(1), logs.astype(np.int64))
    offs = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    return [(int(o), int(g), int(d)) for o, g, d in zip(offs, logs, dirs)], int(sizes.sum())


# ---- what a program keeps --------------------------------------------------

_contexts = {}


def _context(case):
    """One context for each precision and window, as a program keeps them."""
    key = (case["prec"], case["hann"])
    if key not in _contexts:
        c = gbfft.Context(0)
        c.set_precision(case["prec"])
        if case["hann"]:
            c.set_window(gbfft.WINDOW_HANN)
        _contexts[key] = c
    return _contexts[key]


_executor = []


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    n, b = 1 << case["logn"], case["batch"]
    if case["kind"] == "rows":
        if not _executor:
            _executor.append(gbfft.GpuFft.new())
        s.fft = _executor[0]
        x = _input(case, seed, b, n, "cuda").cpu().numpy()
        s.rows = [r.copy() for r in x]  # separate allocations, as a list of vectors is
        return s
    s.ctx = _context(case)
    s.stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "ragged":
        descs, total = _ragged_set(case)
        s.total = total
        s.x = _input(case, seed, 1, total, "cuda").reshape(-1)
        s.y = torch.empty_like(s.x)
        s.plan = s.ctx.ragged_plan(descs)
        return s
    s.x = _input(case, seed, b, n, "cuda")
    if not case["inplace"]:
        s.y = torch.empty_like(s.x)
        if case["op"] == "both":
            s.z = torch.empty_like(s.x)
    return s


def run(s):
    c = s.case
    if c["kind"] == "rows":
        return s.fft.fft(s.rows) if c["op"] == "fwd" else s.fft.ifft(s.rows)
    if c["kind"] == "ragged":
        s.plan.execute(s.x, s.y, s.total, use_graph=True, stream=s.stream)
        return s.y
    n, b = 1 << c["logn"], c["batch"]
    if c["op"] == "both":
        y, z = (s.x, s.x) if c["inplace"] else (s.y, s.z)
        s.ctx.c2c_device(s.x, y, n, b, gbfft.FORWARD, stream=s.stream)
        s.ctx.c2c_device(y, z, n, b, gbfft.INVERSE, stream=s.stream)
        return [z] if c["inplace"] else [y, z]
    s.ctx.c2c_device(s.x, s.y, n, b, gbfft.FORWARD if c["op"] == "fwd" else gbfft.INVERSE, stream=s.stream)
    return s.y


# ---- what a pass cannot do without -----------------------------------------

def work(case):
    if case["kind"] == "ragged":
        descs, total = _ragged_set(case)
        return {"bytes": 16 * total, "flops": sum(5 * g << g for _, g, _ in descs)}
    samples = case["batch"] << case["logn"]
    passes = 2 if case["op"] == "both" else 1
    return {"bytes": 16 * samples * passes, "flops": 5 * case["logn"] * samples * passes}


# ---- the same in 64 bits ---------------------------------------------------

def _hann(case):
    n = 1 << case["logn"]
    i = torch.arange(n, dtype=torch.float64, device="cuda")
    return 0.5 * (1 - torch.cos(2 * math.pi * i / (n - 1)))


def _dft(case, x, forward):
    x = x.to(torch.complex128)
    if case["hann"]:
        x = x * _hann(case)
    return torch.fft.fft(x, dim=-1) if forward else torch.fft.ifft(x, dim=-1)


def exact(case, seed):
    n, b = 1 << case["logn"], case["batch"]
    if case["kind"] == "ragged":
        descs, total = _ragged_set(case)
        x = _input(case, seed, 1, total, "cuda").reshape(-1)
        out = torch.empty(total, dtype=torch.complex128, device="cuda")
        for o, g, d in descs:
            out[o:o + (1 << g)] = _dft(case, x[o:o + (1 << g)], d == gbfft.FORWARD)
        return out
    x = _input(case, seed, b, n, "cuda")
    if case["kind"] == "rows":
        return list(_dft(case, x, case["op"] == "fwd").cpu().numpy())
    if case["op"] == "both":
        y = _dft(case, x, True)
        z = _dft(case, y, False)
        return [z] if case["inplace"] else [y, z]
    return _dft(case, x, case["op"] == "fwd")
