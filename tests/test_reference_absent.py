"""Building without the reference's sources: nothing of it is compiled, and
that is no error, whether its directory is missing or has nothing in it."""
import pytest

from oracle import refrun


@pytest.mark.parametrize("made", [False, True], ids=["no directory", "empty directory"])
def test_the_reference_kernels_are_left_out_without_their_sources(tmp_path, monkeypatch, made):
    where = tmp_path / "reference"
    if made:
        where.mkdir()
    monkeypatch.setattr(refrun, "REFERENCE", str(where))
    monkeypatch.setattr(refrun, "REF_OUT", str(tmp_path / "out"))
    assert refrun.build_cubins() is False
