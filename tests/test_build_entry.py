"""build() without a reference checkout: no folder, or one without the reference's sources."""
import subprocess

import pytest

import __graft_entry__ as entry


@pytest.mark.parametrize("folder", ["absent", "empty"])
def test_build_without_the_reference(monkeypatch, tmp_path, folder):
    ref = tmp_path / folder
    if folder == "empty":
        ref.mkdir()
    made = []
    monkeypatch.setattr(entry, "REF", str(ref))
    monkeypatch.setattr("tmc_gb300.build.build", lambda: made.append("library"))
    monkeypatch.setattr(subprocess, "run", lambda cmd, **kw: made.append(cmd[-1]))
    entry.build()
    assert made == ["library", "liboracle.so"]
