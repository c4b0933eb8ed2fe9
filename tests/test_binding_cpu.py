"""A native binding that is missing, does not load or was built for another torch leaves the ctypes call in its place."""
from __future__ import annotations

import shutil

import pytest


@pytest.fixture
def runtime(monkeypatch):
    from marmot_b200 import runtime

    monkeypatch.setattr(runtime, "_binding", None)
    return runtime


def test_missing_and_broken_modules(runtime, monkeypatch, tmp_path):
    monkeypatch.setattr(runtime, "LIB_PATH", tmp_path / runtime.LIB_PATH.name)
    assert runtime.load_binding() is False
    runtime._binding = None
    (tmp_path / "_binding.so").write_bytes(b"not a library")
    assert runtime.load_binding() is False


def test_another_torch(runtime, monkeypatch, tmp_path):
    import torch
    from marmot_b200 import build

    build.build()
    shutil.copy(build.build_binding(), tmp_path / "_binding.so")
    monkeypatch.setattr(runtime, "LIB_PATH", tmp_path / runtime.LIB_PATH.name)
    monkeypatch.setattr(torch, "__version__", "1.0.0")
    assert runtime.load_binding() is False


def test_the_build_follows_torch(monkeypatch):
    import subprocess

    import torch
    from marmot_b200 import build

    build.build_binding()

    def no_compiler(*a, **k):
        raise AssertionError("compiled again")

    with monkeypatch.context() as m:
        m.setattr(subprocess, "run", no_compiler)
        build.build_binding()  # up to date
        m.setattr(torch, "__version__", "1.0.0")
        with pytest.raises(AssertionError, match="compiled again"):
            build.build_binding()
