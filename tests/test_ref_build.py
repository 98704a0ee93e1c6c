"""The reference's cubins are built only where its sources are: an absent or empty
directory is no error."""
import pytest


@pytest.mark.parametrize("make", [False, True])
def test_no_sources_no_build(tmp_path, monkeypatch, make):
    from oracle import ref_build

    ref = tmp_path / "reference"
    if make:
        ref.mkdir()
    monkeypatch.setattr(ref_build, "REF", str(ref))
    monkeypatch.setattr(ref_build, "OUT", str(tmp_path / "out"))
    assert not ref_build.available()
    assert ref_build.build() == []
