"""The extension behind the hot shims is used only where it belongs to the library beside it."""

from __future__ import annotations

import sys
from types import SimpleNamespace

import pytest
import torch

import lite_llama_b200
from lite_llama_b200 import build
from lite_llama_b200.kernels import _native


@pytest.fixture
def elsewhere(tmp_path, monkeypatch):
    monkeypatch.setattr(build, "FAST_OUT", tmp_path / "_fast.so")
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path)
    return tmp_path


@pytest.mark.parametrize("compiler", ["false", "no-such-compiler"])
def test_an_extension_that_cannot_be_rebuilt_does_not_stay(elsewhere, monkeypatch, compiler):
    for name in ("_fast.so", "fast_calls.stamp"):
        (elsewhere / name).write_text("of an earlier build")
    monkeypatch.setenv("CXX", compiler)
    assert build.build_fast()
    assert list(elsewhere.iterdir()) == []


def test_an_extension_of_another_build_is_not_used(monkeypatch):
    def init(*_):
        raise AssertionError("called")

    for tag in (None, torch.__version__, build.fast_tag("0.0")):
        other = SimpleNamespace(built_for=tag, torch_version=torch.__version__, init=init)
        monkeypatch.setitem(sys.modules, "lite_llama_b200._fast", other)
        monkeypatch.setattr(lite_llama_b200, "_fast", other, raising=False)
        assert _native._table() == {}


def test_the_tag_follows_the_header_and_the_source(tmp_path, monkeypatch):
    tag = build.fast_tag("1")
    for name in ("HEADER", "FAST_SRC"):
        with monkeypatch.context() as m:
            other = tmp_path / name
            other.write_bytes(getattr(build, name).read_bytes() + b" ")
            m.setattr(build, name, other)
            assert build.fast_tag("1") != tag
    assert build.fast_tag("2") != tag
