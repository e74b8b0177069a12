"""The build entry point rebuilds the oracle's pin only from a reference tree
that is there: a missing or an empty directory is passed over.
"""
import os
import subprocess

import pytest


@pytest.mark.parametrize("tree", ["missing", "empty", "sources"])
def test_reference_tree(engine, monkeypatch, tmp_path, tree):
    import __graft_entry__ as entry

    ref = tmp_path / "reference"
    if tree != "missing":
        ref.mkdir()
    if tree == "sources":
        os.makedirs(ref / "origin" / "GoldenC" / "src")
    calls = []
    monkeypatch.setattr(entry, "REFERENCE", str(ref))
    monkeypatch.setattr(subprocess, "run", lambda cmd, **kw: calls.append(cmd))
    entry.build()
    pins = [c for c in calls if any(str(a).endswith("ref.mk") for a in c)]
    assert len(calls) - len(pins) == 2  # the engine and the oracle
    assert len(pins) == (tree == "sources")
