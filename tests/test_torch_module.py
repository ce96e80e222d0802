"""The module built against torch (build.py, native.torch_module): tied to one torch, and not needed by the kernels. No GPU."""
import subprocess

import pytest
import torch

from ccfuser_b200 import build
from ccfuser_b200 import native as N


@pytest.fixture
def untried(monkeypatch):
    monkeypatch.setattr(N, "_torch_module", None)
    monkeypatch.setattr(N, "_torch_module_tried", False)


def test_a_module_of_another_torch_is_not_this_ones(monkeypatch):
    N.load()
    build.build()
    path = build.torch_path()
    assert not build.needs_torch_module()
    monkeypatch.setattr(torch, "__version__", "0.0.0+other")
    assert build.torch_path() != path and build.needs_torch_module()
    assert not build.needs_build()          # the CUDA library is nobody's version


def test_without_a_compiler_the_library_loads_and_nothing_is_built_again(monkeypatch, untried):
    N.load()
    monkeypatch.setattr(torch, "__version__", "0.0.0+other")
    ran = []

    def no_compiler(cmd, *a, **k):
        ran.append(cmd[0])
        raise FileNotFoundError("g++")
    monkeypatch.setattr(subprocess, "check_call", no_compiler)
    monkeypatch.setattr(subprocess, "Popen", no_compiler)
    with pytest.warns(UserWarning, match="LayerNorm"):
        assert N.torch_module() is None
    assert N.torch_module() is None         # tried once
    assert ran == ["g++"] and not build.needs_build()


def test_the_module_of_this_torch_loads(untried):
    assert N.torch_module().launches() >= 0
