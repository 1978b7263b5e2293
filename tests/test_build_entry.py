"""build() makes the reference checker only where the reference's sources are:
an empty directory of that name is no reason to fail."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import __graft_entry__ as entry  # noqa: E402


@pytest.mark.parametrize("sources", [False, True])
def test_reference_build_needs_its_sources(tmp_path, monkeypatch, sources):
    if sources:
        (tmp_path / "hydro_solver_3d.c").write_text("")
    made = []
    monkeypatch.setattr(entry, "REFERENCE", str(tmp_path))
    monkeypatch.setattr(entry, "_make", made.append)
    entry.build()
    assert any("ref" in m for m in made) == sources
