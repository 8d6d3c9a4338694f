"""CPU: the native module is bound to torch's and CPython's ABI, so another version of either rebuilds it."""
import importlib.metadata

import pytest

from dadgpt_b200 import build


@pytest.fixture
def built(monkeypatch):
    build.build()
    calls = []
    monkeypatch.setattr(build, "_build_native", calls.append)
    return calls


def test_a_module_of_this_torch_is_kept(built):
    build.build()
    assert not built


def test_another_torch_rebuilds_the_module(built, monkeypatch):
    monkeypatch.setattr(importlib.metadata, "version", lambda name: "0.0.1")
    build.build()
    assert len(built) == 1


def test_a_module_without_a_record_is_rebuilt(built, monkeypatch, tmp_path):
    monkeypatch.setattr(build, "NATIVE_ABI", str(tmp_path / "none"))
    build.build()
    assert len(built) == 1
