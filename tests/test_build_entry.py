"""build() where the folder of the reference checkout is there but holds no checkout. CPU only."""
import __graft_entry__ as entry
from baseline import stage


def test_build_without_a_checkout(tmp_path, monkeypatch):
    monkeypatch.delenv("LETTUCE_REF", raising=False)
    monkeypatch.setattr(entry, "REFERENCE_CHECKOUT", str(tmp_path))
    monkeypatch.setattr(stage, "STAGE", str(tmp_path / "staged"))
    entry.build()
    assert stage.staged_root() is None
