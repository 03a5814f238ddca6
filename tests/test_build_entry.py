"""The build entry point on a machine without the reference's sources."""
import os

import pytest

import __graft_entry__ as entry


@pytest.mark.parametrize("there", ["nothing", "empty", "sources"])
def test_reference_checker_is_built_from_sources_only(nm, tmp_path, monkeypatch, there):
    ref = tmp_path / "reference"
    if there != "nothing":
        ref.mkdir()
    if there == "sources":
        (ref / "common.cpp").write_text("")
    ran = []
    monkeypatch.setattr(entry, "REFERENCE", os.fspath(ref))
    monkeypatch.setattr(entry, "_run", ran.append)
    entry.build()
    assert any("nested-risk-mlmc_b200" in a for a in ran[0])
    assert sum("ref" in cmd for cmd in ran) == (there == "sources")
