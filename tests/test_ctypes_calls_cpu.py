"""Without the extension module for the installed torch the calls go through ctypes, with a warning."""
import importlib

import pytest

pkg = importlib.import_module("jax-gcm_b200")
L = pkg._lib
build = importlib.import_module("jax-gcm_b200.build")


@pytest.mark.parametrize("broken", [False, True])
def test_missing_or_broken_module(monkeypatch, tmp_path, broken):
    path = tmp_path / "_calls.so"
    if broken:
        path.write_bytes(b"no shared object")
    monkeypatch.setattr(build, "calls_path", lambda: str(path))
    monkeypatch.setattr(L, "_calls", None)
    with pytest.warns(RuntimeWarning, match="ctypes"):
        mod = L.calls()
    assert mod.__name__.endswith("ctypes_calls") and L.calls() is mod


def test_every_native_call_is_there():
    names = [n for n in dir(L.calls()) if not n.startswith("_") and n != "bind"]
    mod = importlib.import_module("jax-gcm_b200.ctypes_calls")
    assert names and all(callable(getattr(mod, n, None)) for n in names)
