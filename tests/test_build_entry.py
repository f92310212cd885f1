"""build() without the reference's sources: an empty or missing reference folder leaves
the oracle binaries out instead of failing."""
import importlib
import subprocess

import pytest


@pytest.mark.parametrize("present", ["missing", "empty", "sources"])
def test_oracle_only_with_sources(tmp_path, monkeypatch, present):
    import __graft_entry__ as entry
    ref = tmp_path / "reference"
    if present != "missing":
        ref.mkdir()
    if present == "sources":
        (ref / "src").mkdir()
        (ref / "src" / "pmx.cpp").write_text("")
    monkeypatch.setenv("PMX_REFERENCE_DIR", str(ref))
    monkeypatch.setattr(subprocess, "run", lambda cmd, **kw: calls.append(cmd))
    calls = []
    entry = importlib.reload(entry)
    try:
        entry.build()
    finally:
        monkeypatch.delenv("PMX_REFERENCE_DIR")
        importlib.reload(entry)
    assert sum("oracle" in " ".join(c) for c in calls) == (present == "sources")
