"""CPU tests of the build: the library does not depend on the extension."""
import sys

import pytest

torch = pytest.importorskip("torch")

from relax_b200 import build


def test_the_library_is_built_without_torch(monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", None)                 # (import torch raises ImportError)
    assert build.build() == build.LIB


@pytest.mark.parametrize("command", [["/bin/sh", "-c", "echo no such header; exit 1"], ["/no/such/compiler"]])
def test_a_failed_extension_costs_the_extension_only(monkeypatch, command):
    monkeypatch.setattr(build, "_torch_call_command", lambda *_: command)
    monkeypatch.setattr(build, "_torch_call_stale", lambda *_: True)
    with pytest.warns(RuntimeWarning, match="(?i)no such"):
        assert build.build() == build.LIB
