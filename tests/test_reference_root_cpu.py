"""Where gsbn's source tree is looked for: an empty folder in its place is no
tree, so the tests that read its files are skipped and do not fail."""
from oracle import sim


def test_reference_root(tmp_path, monkeypatch):
    monkeypatch.setenv("GSBN_REFERENCE_ROOT", str(tmp_path))
    assert sim.reference_root() is None
    (tmp_path / "data").mkdir()
    assert sim.reference_root() == str(tmp_path)
    monkeypatch.setenv("GSBN_REFERENCE_ROOT", str(tmp_path / "none"))
    assert sim.reference_root() is None
