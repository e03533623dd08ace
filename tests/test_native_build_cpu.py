"""The CUDA library does not depend on the extension module of the native host path: it builds and loads without it, and a
module built for another torch or Python is never taken."""
import subprocess

import pytest
import torch

from bitmtp_b200 import native


@pytest.fixture
def unloaded(monkeypatch):
    """lib() starts afresh, and what it sets is put back."""
    monkeypatch.setattr(native, "_lib", None)
    monkeypatch.setattr(native, "_host", None)
    return monkeypatch


def test_the_library_loads_with_the_module(unloaded):
    assert native.lib() is not None and native._host is not None
    assert native._host.linear() is None and native._host.linear_rows() is None


@pytest.mark.parametrize("content", [None, b"not an object file"])
def test_the_library_loads_without_the_module(unloaded, tmp_path, content):
    so = tmp_path / "_host.so"
    if content is not None:
        so.write_bytes(content)
    unloaded.setattr(native, "host_so_path", lambda: str(so))
    with pytest.warns(RuntimeWarning, match="no native host path"):
        assert native.lib().bm_t2_gemv_bytes(1, 6144, 2048, 0) == 3356676
    assert native._host is None


def test_another_torch_or_python_has_a_module_of_its_own(monkeypatch):
    here = native.host_so_path()
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    other = native.host_so_path()
    monkeypatch.setattr(native.sysconfig, "get_config_var", lambda name: "cpython-399")
    assert len({here, other, native.host_so_path()}) == 3


def test_the_library_is_built_first_and_without_the_modules_compiler(monkeypatch, tmp_path):
    ran = []

    def run(cmd, check):
        ran.append(cmd[0])
        if cmd[0] != "the-nvcc":
            raise FileNotFoundError(cmd[0])
        (tmp_path / "lib.so.tmp").write_bytes(b"built")

    monkeypatch.setenv("NVCC", "the-nvcc")
    monkeypatch.setenv("CXX", "no-such-compiler")
    monkeypatch.setattr(subprocess, "run", run)
    monkeypatch.setattr(native, "SO_PATH", str(tmp_path / "lib.so"))
    monkeypatch.setattr(native, "host_so_path", lambda: str(tmp_path / "_host.so"))
    assert native.build(force=True) == str(tmp_path / "lib.so")
    assert ran == ["the-nvcc", "no-such-compiler"] and (tmp_path / "lib.so").read_bytes() == b"built"
