"""CPU: the extension module beside the library (gbfft/_call.c) is of use, or absent: one
that cannot be built or loaded leaves the library and its ctypes calls as they are."""
import importlib
import os
import shutil
import sysconfig

import pytest


@pytest.fixture
def build_module(monkeypatch, tmp_path):
    import gbfft
    b = importlib.import_module(gbfft.build.__module__)
    monkeypatch.setattr(b, "CALL_PATH", str(tmp_path / os.path.basename(b.CALL_PATH)))
    return b


def test_name_is_this_interpreters(build_module):
    assert os.path.basename(build_module.CALL_PATH) == "_gbfft_call" + sysconfig.get_config_var("EXT_SUFFIX")


@pytest.mark.parametrize("cc", [shutil.which("false"), "/no/such/compiler"])
def test_a_compiler_that_fails_is_a_warning(build_module, monkeypatch, cc):
    if not os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")):
        pytest.skip("no Python headers")
    open(build_module.CALL_PATH, "w").close()  # what an older source left
    monkeypatch.setenv("CC", cc)
    with pytest.warns(UserWarning, match="_call.c"):
        build_module._build_call(True)
    assert not os.path.exists(build_module.CALL_PATH)


def test_a_compiler_with_arguments(build_module, monkeypatch):
    if not shutil.which("gcc") or not os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")):
        pytest.skip("no gcc or Python headers")
    monkeypatch.setenv("CC", "gcc -O1")
    build_module._build_call(True)
    assert os.path.getsize(build_module.CALL_PATH) > 0


def test_a_module_that_does_not_load(lib_built, monkeypatch, tmp_path):
    from gbfft import _lib
    bad = tmp_path / "_gbfft_call.so"
    bad.write_bytes(b"not a shared object")
    for name, value in (("_lib", None), ("_c2c", None), ("CALL_PATH", str(bad))):
        monkeypatch.setattr(_lib, name, value)
    assert _lib.load().gbfft_version()
    assert _lib._c2c is None
