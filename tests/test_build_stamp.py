"""The stamp that decides whether the built libraries are current covers what the host library is compiled against (PyTorch, its
CUDA, its C++ ABI and the Python ABI): a library built for another PyTorch counts as stale."""

import sysconfig

import pytest
import torch

from fms_model_optimizer_b200 import build_ext


@pytest.mark.parametrize("what", ["torch", "cuda", "cxx11", "python"])
def test_another_environment_makes_the_build_stale(monkeypatch, tmp_path, what):
    for name in ("LIB_PATH", "HOST_PATH", "STAMP_PATH"):
        path = tmp_path / name
        path.write_text(build_ext.source_digest() + "\n")
        monkeypatch.setattr(build_ext, name, path)
    assert not build_ext.is_stale()
    if what == "torch":
        monkeypatch.setattr(torch, "__version__", "0.0.1")
    elif what == "cuda":
        monkeypatch.setattr(torch.version, "cuda", "0.1")
    elif what == "cxx11":
        monkeypatch.setattr(torch._C, "_GLIBCXX_USE_CXX11_ABI", not torch._C._GLIBCXX_USE_CXX11_ABI)
    else:
        get = sysconfig.get_config_var
        monkeypatch.setattr(sysconfig, "get_config_var", lambda name: "cpython-00" if name == "SOABI" else get(name))
    assert build_ext.is_stale()
