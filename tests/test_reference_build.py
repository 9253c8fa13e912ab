"""The reference build is skipped where its source tree is absent or empty."""
from oracle import bindings


def test_empty_reference_tree_is_no_build_error(tmp_path, monkeypatch):
    monkeypatch.setattr(bindings, "REF_SO", str(tmp_path / "libhyowon_ref.so"))
    assert bindings.build_reference(str(tmp_path)) is False
    assert bindings.build_reference(str(tmp_path / "absent")) is False
