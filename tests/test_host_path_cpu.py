"""The native host path is an accelerator, not a requirement: without it, or with one built for another torch or Python, launches
go through the Python checks; and the build notices both.  No GPU."""
import importlib
import types

import pytest


@pytest.fixture
def ffi(pkg, monkeypatch):
    m = importlib.import_module("glm53f-afd_b200.ffi")
    monkeypatch.setattr(m, "_native", None)
    return m


def takes_no_call(host):
    return host.core_decode(*[None] * 18) == -1 and host.chain_batch(None, None, None, False) == -1 and host.raw_stream(None) is None


def test_without_the_module(ffi, monkeypatch, tmp_path):
    monkeypatch.setattr(ffi._build, "HOST", str(tmp_path / "_host.so"))
    with pytest.warns(RuntimeWarning, match="is missing"):
        assert takes_no_call(ffi.host())
    assert takes_no_call(ffi.host())
    assert ffi._build._host_stale(ffi._build.HOST)


@pytest.mark.parametrize("other", ["torch 1.0, python 3.12", "torch 2.11.0+cu128, python 2.7"])
def test_with_a_module_built_for_something_else(ffi, monkeypatch, tmp_path, other):
    built = tmp_path / "_host.so"
    built.write_bytes(b"\0" + other.encode() + b"\0")
    monkeypatch.setattr(ffi._build, "HOST", str(built))
    monkeypatch.setattr(importlib.import_module("glm53f-afd_b200"), "_host", types.SimpleNamespace(built_for=other), raising=False)
    with pytest.warns(RuntimeWarning, match="built for"):
        assert takes_no_call(ffi.host())
    monkeypatch.setattr(ffi._build, "_stale", lambda *_: False)
    assert ffi._build._host_stale("")
    built.write_bytes(b"\0" + ffi._build.host_built_for().encode() + b"\0")
    assert not ffi._build._host_stale("")


def test_the_built_module_is_taken(ffi):
    h = ffi.host()
    assert h.built_for == ffi._build.host_built_for() and h.core_decode(*[None] * 18) == -1
