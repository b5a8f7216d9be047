"""Loading of the host extension: what happens where it cannot be had."""
import importlib.util
import warnings

import pytest
import torch

from maxdiffusion_b200 import build
from maxdiffusion_b200.ops import _lib


@pytest.fixture
def fresh(monkeypatch, tmp_path):
  """A GPU machine, as far as the loader can see, with an empty folder in place of the package's."""
  monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
  monkeypatch.setattr(_lib, "lib", lambda: None)
  monkeypatch.setattr(_lib, "_HOST", None)
  monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "_kernels.so")
  monkeypatch.delenv("MDB200_NO_AUTOBUILD", raising=False)
  return tmp_path


def _object(built_for):
  return b"not a shared object \0mdb_host_ops built for " + built_for.encode() + b";\0"


def test_the_object_says_what_it_was_built_for(tmp_path):
  if build.HOST_PATH.exists():
    assert build.host_ops_built_for(build.HOST_PATH) == build.host_ops_target()
  assert build.host_ops_built_for(tmp_path / "none.so") is None


def _takes_nothing():
  with pytest.warns(RuntimeWarning, match="host extension"):
    host = _lib.host_ops()
  assert host.linear(1, 2) is NotImplemented and host.conv() is NotImplemented and host.launches() == 0
  with warnings.catch_warnings():
    warnings.simplefilter("error")
    assert _lib.host_ops() is host  # said once
  assert _lib.launch_count() == _lib._launches


def test_missing_and_not_to_be_built(fresh, monkeypatch):
  monkeypatch.setenv("MDB200_NO_AUTOBUILD", "1")
  _takes_nothing()


def test_a_machine_that_cannot_compile_it(fresh, monkeypatch):
  def fail(*a, **k):
    raise RuntimeError("host_ops.cpp: g++ failed")
  monkeypatch.setattr(build, "build_host_ops", fail)
  _takes_nothing()


def test_no_compiler_at_all(fresh, monkeypatch):
  def fail(*a, **k):
    raise FileNotFoundError("g++")
  monkeypatch.setattr(build, "build_host_ops", fail)
  _takes_nothing()


def test_an_object_that_does_not_load(fresh):
  (fresh / "_host_ops.so").write_bytes(_object(build.host_ops_target()))
  _takes_nothing()


@pytest.mark.parametrize("built_for", [None, "PyTorch 2.0.0, Python 3.8.1"])
def test_an_object_for_another_pytorch_is_rebuilt_and_not_loaded(fresh, monkeypatch, built_for):
  (fresh / "_host_ops.so").write_bytes(b"an object" if built_for is None else _object(built_for))
  asked, load = [], importlib.util.spec_from_file_location

  def refuse(name, *a, **k):
    assert name != "_host_ops", "loaded"
    return load(name, *a, **k)
  monkeypatch.setattr(importlib.util, "spec_from_file_location", refuse)

  def fail(*a, **k):
    asked.append(1)
    raise RuntimeError("no compiler")
  monkeypatch.setattr(build, "build_host_ops", fail)
  _takes_nothing()
  assert asked == [1]
  monkeypatch.setenv("MDB200_NO_AUTOBUILD", "1")
  monkeypatch.setattr(_lib, "_HOST", None)
  _takes_nothing()
  assert asked == [1]
