"""The host path is found only by the torch, the Python and the source it was built for."""
import os
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
