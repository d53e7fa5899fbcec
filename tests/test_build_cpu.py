"""The native host side of eager calls is built for one Python and torch, and is optional."""
import pytest
import torch

from sparser_faster_llms_b200 import build, twell


def test_the_module_of_another_torch_is_not_loaded(monkeypatch):
    own = build.host_path()
    assert torch.__version__ in own.name
    build.build_library()
    assert own.exists() and twell._load_host_call() is not None
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.host_path() != own and twell._load_host_call() is None


def test_a_failed_host_build_leaves_the_library(monkeypatch, tmp_path):
    bad = tmp_path / "host_call.cpp"
    bad.write_text("#error no host module\n")
    build.build_library()
    monkeypatch.setattr(build, "HOST_SOURCE", bad)
    monkeypatch.setattr(build, "host_path", lambda: tmp_path / "_host_call.so")
    with pytest.warns(UserWarning, match="no host module"):
        assert build.build_library() == build.LIB_PATH
    assert list(tmp_path.iterdir()) == [bad]


def test_without_a_compiler_the_library_stays(monkeypatch, tmp_path):
    build.build_library()
    monkeypatch.setattr(build, "host_path", lambda: tmp_path / "_host_call.so")
    monkeypatch.setattr(build.shutil, "which", lambda name: None if name != "nvcc" else "/usr/bin/nvcc")
    monkeypatch.setenv("PATH", str(tmp_path))
    with pytest.warns(UserWarning, match="not built"):
        assert build.build_library() == build.LIB_PATH


def test_a_module_that_does_not_load_is_said_once_and_left_out(monkeypatch, tmp_path):
    broken = tmp_path / "_host_call.so"
    broken.write_bytes(b"not a library")
    monkeypatch.setattr(build, "host_path", lambda: broken)
    with pytest.warns(UserWarning, match="does not load"):
        assert twell._load_host_call() is None
