"""build() without the reference checkout: a directory that is there but empty is no checkout."""
import os
import sys

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_empty_reference_directory(tmp_path, monkeypatch):
    monkeypatch.syspath_prepend(REPO)
    sys.modules.pop("__graft_entry__", None)
    import __graft_entry__ as g

    monkeypatch.setattr(g, "REFERENCE", str(tmp_path))
    assert not g.has_reference(str(tmp_path))
    g.build()
    (tmp_path / "source").mkdir()
    (tmp_path / "source" / "multipole_expansion.cc").write_text("")
    assert g.has_reference(str(tmp_path))
