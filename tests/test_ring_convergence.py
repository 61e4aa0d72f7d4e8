"""CPU: the ring kernels meet at whole-warp barriers with whole warps.

`bar.sync`, and `__syncthreads()`, are a warp's: every lane of it arrives together.  The
loader's and the storer's role is one lane's, and lanes without a transform skip a rows
tile's loads and stores, so a `__syncwarp()` stands before the barrier that follows."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "wgls-rs-fft_gb300", "csrc")


def _statements(path, start):
    """The statements of the function that begins at `start`, without comments."""
    text = open(os.path.join(CSRC, path)).read()
    text = re.sub(r"//[^\n]*|^#[^\n]*$", "", text[text.index(start):], flags=re.M)
    depth = 0
    for i in range(text.index("{"), len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            break
    return [" ".join(s.split()) for s in re.split(r"[;{}]", text[:i]) if s.strip()]


@pytest.mark.parametrize("path,kernel,finish", [("fft_pipe.cuh", "fft_pipe_kernel(", "fused_finish"),
                                                ("fft_ragged_pipe.cu", "fft_ragged_pipe_kernel(", "rag_finish")])
def test_roles_reconverge_before_the_closing_barrier(path, kernel, finish):
    st = _statements(path, kernel)
    last_role = max(i for i, s in enumerate(st) if "_storer" in s)
    close = next(i for i in range(last_role, len(st)) if st[i].startswith(("__syncthreads", finish)))
    assert st[close - 1] == "__syncwarp()", st[close - 2:close + 1]


def test_group_barrier_is_a_whole_warps():
    st = _statements("fft_tiles.cuh", "void tile_sync(")
    bar = next(i for i, s in enumerate(st) if "bar.sync" in s)
    assert "__syncwarp()" in st[:bar], st
