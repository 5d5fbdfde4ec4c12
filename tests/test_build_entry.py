"""build() where the reference's sources are not at hand."""
import subprocess

import pytest


@pytest.mark.parametrize("present", [False, True])
def test_build_without_reference_sources(monkeypatch, tmp_path, present):
    """A missing or an empty reference directory leaves its targets out."""
    import __graft_entry__ as entry
    from culbm_b200 import build as native
    ref = tmp_path / "reference"
    if present:
        ref.mkdir()
    monkeypatch.setattr(entry, "REFERENCE", str(ref))
    monkeypatch.setattr(native, "build", lambda: None)
    run, calls = subprocess.run, []

    def record(cmd, *args, **kw):
        calls.append(cmd)
        return run(cmd, *args, **kw)

    monkeypatch.setattr(subprocess, "run", record)
    entry.build()
    assert calls and not any("ref-cpu" in c or "ref-gpu" in c for c in calls)
