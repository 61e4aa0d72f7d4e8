"""CPU: the index maps of the warp-column tiles (fft_warp.cuh) against a model of
the tensor-map swizzle, their in-warp exchange and bank conflicts, and the
two-column butterflies (fft_pair.cuh) against the single-column ones, compiled
for the host by nvcc from the kernels' own functions (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "cpp", "warp_tiles.cu")
CSRC = os.path.join(ROOT, "wgls-rs-fft_gb300", "csrc")


def test_warp_tiles(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "warp_tiles")
    r = subprocess.run([nvcc, "-std=c++20", "--expt-relaxed-constexpr", "-Xcompiler", "-ffp-contract=off",
                        "-I", os.path.join(ROOT, "include"), "-I", CSRC, SRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    tiles = [tuple(int(v) for v in line.split()[1:]) for line in out if line.startswith("tile ")]
    dfts = [tuple(int(v) for v in line.split()[1:]) for line in out if line.startswith("dft ")]
    assert len(tiles) == 7 and len(dfts) == 4
    for kind, logr, logtile, ok, conflicts in tiles:
        assert ok == 1, (kind, logr, logtile)
        # one column a thread: a radix-2^10 column fills a warp, which then reads one half
        # of every chunk
        assert conflicts == (2 if kind == 5 and logr == 10 else 1), (kind, logr, conflicts)
    for radix, ok in dfts:
        assert ok == 1, radix
