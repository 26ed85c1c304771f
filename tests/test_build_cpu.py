"""The host path is found only by the torch, the Python and the source it was built for."""
import os
import shutil
import subprocess
import sys
import sysconfig

import pytest
import torch

from void_b200 import _lib, build


def test_the_name_of_the_host_path_follows_what_it_depends_on(monkeypatch, tmp_path):
    _lib.native()
    path = build.native_path()
    assert os.path.exists(path) and not build.needs_build()
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0.0")
        assert build.native_path() != path and build.needs_build()
    with monkeypatch.context() as m:
        m.setattr(sysconfig, "get_config_var", lambda name: "cpython-399-x86_64-linux-gnu")
        assert build.native_path() != path and build.needs_build()
    with monkeypatch.context() as m:
        source = tmp_path / "host.cpp"
        source.write_text(open(build.HOST_SOURCE).read() + "\n")
        m.setattr(build, "HOST_SOURCE", str(source))
        assert build.native_path() != path and build.needs_build()
    assert build.native_path() == path


def test_a_host_path_built_for_something_else_is_not_loaded(monkeypatch):
    _lib.load()
    monkeypatch.setattr(_lib, "_NATIVE", None)
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    with pytest.raises(_lib.VoidB200Error, match="missing"):
        _lib.native()


def test_a_copied_package_runs_its_own_kernels(tmp_path):
    """The host path loads the library beside it, wherever the two were built."""
    _lib.native()
    native, library = (shutil.copy(p, tmp_path) for p in (build.native_path(), build.LIB_PATH))
    code = """
import importlib.util, torch
spec = importlib.util.spec_from_file_location("void_b200._native", %r)
importlib.util.module_from_spec(spec)
print([l.split()[-1] for l in open("/proc/self/maps") if "libvoid_b200.so" in l][0])
""" % native
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == library
