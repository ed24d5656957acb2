"""The oracle's build on machines with and without the reference's sources."""
import pytest

from oracle import stage_ref


def test_an_empty_default_checkout_is_no_checkout(monkeypatch, tmp_path):
    """An empty directory at the default location stages nothing (and the
    restatement still builds); one with the sources is used."""
    monkeypatch.delenv("CONSTRAINTPHYSICS_REFERENCE", raising=False)
    monkeypatch.setattr(stage_ref, "DEFAULT_REFERENCE_ROOT", str(tmp_path))
    assert stage_ref.reference_root() is None
    for d in stage_ref.source_dirs(str(tmp_path)):
        (tmp_path / d).mkdir(parents=True)
    assert stage_ref.reference_root() == str(tmp_path)


def test_a_named_checkout_without_sources_is_refused(monkeypatch, tmp_path):
    monkeypatch.setenv("CONSTRAINTPHYSICS_REFERENCE", str(tmp_path))
    assert stage_ref.reference_root() == str(tmp_path)
    with pytest.raises(SystemExit):
        stage_ref.stage(str(tmp_path))
