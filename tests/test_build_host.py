"""The build's own bookkeeping (nothing is compiled here)."""
from __future__ import annotations

import importlib.metadata

import pytest

from racetrack_b200 import _lib, build


@pytest.fixture
def other_torch(monkeypatch):
    monkeypatch.setattr(importlib.metadata, "version", lambda name: "0.0.0+other")


def test_another_torch_is_another_build(request):
    before = build._fingerprint()
    assert build._fingerprint() == before
    request.getfixturevalue("other_torch")
    assert build._fingerprint() != before


def test_a_module_of_another_torch_is_not_loaded(other_torch, monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_native", None)
    stamp = tmp_path / "_rt_torch.stamp"
    stamp.write_text("torch 1.0 python 3.12")
    monkeypatch.setattr(_lib, "TORCH_STAMP", stamp)
    with pytest.raises(RuntimeError, match="built for torch 1.0"):
        _lib.native()
