"""build() where the place of the reference's sources is absent, or there and empty."""

import importlib

import pytest


@pytest.mark.parametrize("there", [False, True])
def test_build_without_reference_sources(tmp_path, monkeypatch, there):
    entry = importlib.import_module("__graft_entry__")
    tree = tmp_path / "reference"
    if there:
        tree.mkdir()
    monkeypatch.setattr(entry, "REFERENCE_TREE", str(tree))
    called = []
    monkeypatch.setattr("qlat_b200.build.build", lambda: called.append("library"))
    monkeypatch.setattr("oracle.oracle.build", lambda: called.append("oracle"))
    entry.build()
    assert called == ["library", "oracle"]
