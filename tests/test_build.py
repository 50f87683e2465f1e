"""CPU tests of the build script's choices: a host without torch gets the library, and the native host path is built again
after torch has changed."""
import importlib.util
import os
import subprocess
import types

import pytest

from conftest import ROOT


@pytest.fixture
def build(monkeypatch, tmp_path):
    spec = importlib.util.spec_from_file_location("srwm_build", os.path.join(ROOT, "modern-srwm_b200", "csrc", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    monkeypatch.setattr(mod, "_build", lambda *a: "library")
    monkeypatch.setattr(mod, "OBJ", str(tmp_path / "build"))
    monkeypatch.setattr(mod, "HOST", str(tmp_path / "_host.so"))
    return mod


def test_a_host_without_torch_builds_the_library_alone(build, monkeypatch):
    def none(*a):
        raise AssertionError("the native host path needs torch")
    monkeypatch.setattr(build, "build_host", none)
    find = importlib.util.find_spec
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    assert build.build() == "library"
    monkeypatch.undo()
    monkeypatch.setattr(build, "_build", lambda *a: "library")
    monkeypatch.setattr(build, "build_host", none)
    assert build.build(host=False) == "library"
    with pytest.raises(AssertionError):
        build.build()


def test_the_host_path_is_built_again_after_torch_has_changed(build, monkeypatch):
    runs = []

    def run(cmd, **kw):
        runs.append(cmd)
        open(build.HOST, "w").close()
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")
    monkeypatch.setattr(subprocess, "run", run)
    build.build_host()
    build.build_host()
    assert len(runs) == 1
    monkeypatch.setattr(importlib.import_module("importlib.metadata"), "version", lambda name: "99.0")
    build.build_host()
    build.build_host()
    assert len(runs) == 2
