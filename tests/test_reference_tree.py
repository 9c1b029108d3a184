"""A folder without the reference's sources is no reference tree: nothing tries to build or read them there."""
from oracle import ref_build


def test_folder_without_sources(tmp_path, monkeypatch):
    monkeypatch.setattr(ref_build, "REF", str(tmp_path))
    assert ref_build.reference_tree() is None
    for name in ref_build.PLUGINS:
        (tmp_path / f"{name}.cu").write_text("")
    assert ref_build.reference_tree() == str(tmp_path)
