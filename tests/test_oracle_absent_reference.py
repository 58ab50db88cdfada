"""Without the compiled reference (oracle/_ref) its wrapper can be made, as a test
does before it asks ref_available() and skips; only its use fails."""
import pytest


def test_reference_wrapper_without_the_reference(monkeypatch, tmp_path):
    import oracle as oracle_mod

    monkeypatch.setattr(oracle_mod, "REF_DIR", str(tmp_path))
    assert not oracle_mod.ref_available()
    R = oracle_mod.RefE2G()
    with pytest.raises(OSError):
        R.log()
