"""CPU tests of the build: the library does not depend on the extension, and an extension belongs to one torch and one Python."""
import sys

import pytest

torch = pytest.importorskip("torch")

from relax_b200 import build, ops


def test_the_library_is_built_without_torch(monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", None)                 # (import torch raises ImportError)
    assert build.build() == build.LIB


@pytest.mark.parametrize("command", [["/bin/sh", "-c", "echo no such header; exit 1"], ["/no/such/compiler"]])
def test_a_failed_extension_costs_the_extension_only(monkeypatch, command):
    monkeypatch.setattr(build, "_torch_call_command", lambda *_: command)
    monkeypatch.setattr(build, "_torch_call_stale", lambda *_: True)
    with pytest.warns(RuntimeWarning, match="(?i)no such"):
        assert build.build() == build.LIB


def test_an_extension_of_another_torch_is_neither_fresh_nor_loaded(monkeypatch):
    assert not build._torch_call_stale(build.torch_call_path(torch.__version__))
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".other")
    assert build._torch_call_stale(build.torch_call_path(torch.__version__))
    monkeypatch.setattr(ops, "_native", None)
    assert ops._torch_call() is False
