"""The native host side of the torch-tensor calls is optional: calls work without it, and it is built again for another torch."""
import sys
import warnings
from importlib import metadata

import pytest

from laplace_b200 import build, device


class _Lib:
    def laplace_cuda_init(self, dev):
        return 0


@pytest.fixture
def unbound(monkeypatch):
    import torch
    from laplace_b200 import matmul
    monkeypatch.setattr(device, "_ready_on", None)
    monkeypatch.setattr(device, "_native", None)
    monkeypatch.setattr(matmul, "_initialised", False)
    monkeypatch.setattr(device._lib, "load", _Lib)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)


def test_a_missing_native_module_leaves_the_general_path(unbound, monkeypatch):
    import laplace_b200
    monkeypatch.delattr(laplace_b200, "_native", raising=False)
    monkeypatch.setitem(sys.modules, "laplace_b200._native", None)        # what importing it then raises is ImportError
    with pytest.warns(RuntimeWarning, match="goes through ctypes"):
        assert isinstance(device.lib(), _Lib)
    assert device._native is None and device._ready_on == 0
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        device.lib()                                                      # said once


@pytest.fixture
def commands(monkeypatch, tmp_path):
    seen = []

    def run(cmd, **_):
        seen.append(cmd)
        (tmp_path / "_native.so").write_bytes(b"")
        return type("R", (), {"returncode": 0, "stdout": "", "stderr": ""})()

    monkeypatch.setattr(build, "PKG", tmp_path)
    monkeypatch.setattr(build, "NATIVE", tmp_path / "_native.so")
    monkeypatch.setattr(build.subprocess, "run", run)
    return seen


def test_another_torch_builds_the_module_again(commands, monkeypatch):
    build.build_native()
    build.build_native()
    assert len(commands) == 1
    monkeypatch.setattr(metadata, "version", lambda name: "0.0.1")
    build.build_native()
    build.build_native()
    assert len(commands) == 2


def test_without_torch_the_module_is_left_out(commands, monkeypatch, capsys):
    def missing(name):
        raise metadata.PackageNotFoundError(name)

    monkeypatch.setattr(metadata, "version", missing)
    assert build.build_native() is None and not commands
    assert "left out" in capsys.readouterr().err
