"""The reference build is skipped where its source tree is absent or empty."""
import pytest

from conftest import reference_or_skip
from oracle import bindings


def test_empty_reference_tree_is_no_build_error(tmp_path, monkeypatch):
    monkeypatch.setattr(bindings, "REF_SO", str(tmp_path / "libhyowon_ref.so"))
    assert bindings.build_reference(str(tmp_path)) is False
    assert bindings.build_reference(str(tmp_path / "absent")) is False


def test_fixtures_skip_without_the_reference(tmp_path, monkeypatch):
    """The parity tests' fixtures: a skip, not an error, where nothing can be built."""
    monkeypatch.setattr(bindings, "REF_SO", str(tmp_path / "libhyowon_ref.so"))
    monkeypatch.setenv("HYOWON_REF_ROOT", str(tmp_path))
    with pytest.raises(pytest.skip.Exception):
        reference_or_skip()
