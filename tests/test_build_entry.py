"""build() compiles the reference harness only where the reference's sources are."""
import __graft_entry__ as entry


def test_reference_harness_needs_its_sources(monkeypatch, tmp_path):
    made = []
    monkeypatch.setattr(entry, "_make", lambda path, *extra: made.append(path))
    monkeypatch.setattr(entry, "REFERENCE_DIR", str(tmp_path))  # a folder without sources
    entry.build()
    assert not [p for p in made if p.replace("\\", "/").endswith("oracle/ref")]
    (tmp_path / "GridKNNCuda.cu").write_text("")
    entry.build()
    assert [p for p in made if p.replace("\\", "/").endswith("oracle/ref")]
