"""Build recipe for libgbfft.so (sm_103a only).

Each ``csrc/*.cu`` is compiled by nvcc in parallel, then linked into
``wgls-rs-fft_gb300/lib/libgbfft.so``.  Cross-compiles without a GPU.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shlex
import shutil
import subprocess
import sysconfig
import warnings

PKG_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
REPO_ROOT = os.path.dirname(PKG_ROOT)
CSRC = os.path.join(PKG_ROOT, "csrc")
LIB_DIR = os.path.join(PKG_ROOT, "lib")
OBJ_DIR = os.path.join(PKG_ROOT, "_build")
LIB_PATH = os.path.join(LIB_DIR, "libgbfft.so")
CALL_SRC = os.path.join(PKG_ROOT, "gbfft", "_call.c")
# (the suffix names interpreter and platform: each finds only a module of its own)
CALL_PATH = os.path.join(LIB_DIR, "_gbfft_call" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
INCLUDE = os.path.join(REPO_ROOT, "include")

ARCH_FLAGS = ["-gencode", "arch=compute_103a,code=sm_103a"]
NVCC_FLAGS = ["-std=c++20", "-O3", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-Wall",
              "--expt-relaxed-constexpr"]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the GB300 FFT library cannot be built")


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    hs.append(os.path.join(INCLUDE, "gbfft.h"))
    return hs


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths)


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
    deps = [os.path.join(CSRC, src)] + _headers()
    if os.path.exists(obj) and os.path.getmtime(obj) >= _newest(deps):
        return obj
    cmd = [nvcc(), *ARCH_FLAGS, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        print(r.stderr)
    return obj


def _build_call(force: bool) -> None:
    """The interpreter-side call (``_call.c``); without Python's headers or a C compiler that
    takes it, the binding makes its calls through ctypes."""
    include = sysconfig.get_paths()["include"]
    cc = shlex.split(os.environ.get("CC", "")) or [shutil.which("gcc") or shutil.which("cc")]
    if not cc[0] or not os.path.exists(os.path.join(include, "Python.h")):
        return
    if not force and os.path.exists(CALL_PATH) and os.path.getmtime(CALL_PATH) >= os.path.getmtime(CALL_SRC):
        return
    if os.path.exists(CALL_PATH):
        os.remove(CALL_PATH)  # of an older source
    try:
        r = subprocess.run([*cc, "-O2", "-shared", "-fPIC", "-Wall", "-I", include, "-o", CALL_PATH, CALL_SRC],
                           capture_output=True, text=True)
        why = r.stderr if r.returncode else None
    except OSError as e:
        why = str(e)
    if why is not None:
        warnings.warn(f"{cc[0]} failed on _call.c; c2c_device goes through ctypes:\n{why}")


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile (if stale) and link libgbfft.so; returns its path."""
    os.makedirs(OBJ_DIR, exist_ok=True)
    os.makedirs(LIB_DIR, exist_ok=True)
    srcs = _sources()
    if force:
        for s in srcs:
            o = os.path.join(OBJ_DIR, s[:-3] + ".o")
            if os.path.exists(o):
                os.remove(o)
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
    if force or not os.path.exists(LIB_PATH) or os.path.getmtime(LIB_PATH) < _newest(objs):
        cmd = [nvcc(), *ARCH_FLAGS, "-shared", "-o", LIB_PATH, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_call(force)
    return LIB_PATH


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
