"""build(): the library first and without torch; the extension module after it, under a name that says
what it was built for; a failure there named apart.  Nothing is compiled here."""
import importlib
import subprocess
import sys
import sysconfig
from types import SimpleNamespace

import pytest
import torch

build = importlib.import_module("jax-gcm_b200.build")


@pytest.fixture
def steps(monkeypatch):
    done = []

    def run(cmd, **kw):
        done.append("extension" if any(str(c).endswith("torch_calls.cpp") for c in cmd)
                    else "library")
        return SimpleNamespace(returncode=int(done[-1] == steps_fail["step"]), stdout="", stderr="")

    steps_fail = {"step": None}
    monkeypatch.setattr(subprocess, "run", run)
    monkeypatch.setattr(build.subprocess, "run", run)
    return done, steps_fail


def test_library_first(steps):
    done, _ = steps
    assert build.build(force=True) == build.OUT
    assert done[-1] == "extension" and set(done[:-1]) == {"library"} and len(done) > 2


def test_library_without_torch(steps, monkeypatch, capsys):
    done, _ = steps
    monkeypatch.setitem(sys.modules, "torch", None)
    assert build.build(force=True) == build.OUT
    assert set(done) == {"library"} and "torch" in capsys.readouterr().err


def test_library_with_a_torch_without_cuda(steps, monkeypatch):
    done, _ = steps
    monkeypatch.setattr(torch.version, "cuda", None)
    assert build.build(force=True) == build.OUT
    assert set(done) == {"library"}


def test_failed_extension_is_named(steps):
    done, fail = steps
    fail["step"] = "extension"
    with pytest.raises(RuntimeError, match="the library is built"):
        build.build(force=True)
    assert "library" in done


def test_name_says_torch_cuda_and_interpreter(monkeypatch):
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    a = build.calls_path()
    assert a.endswith(suffix) and torch.__version__ in a
    monkeypatch.setattr(torch, "__version__", "2.11.0+cu130")
    assert build.calls_path() != a and "cu130" in build.calls_path()
