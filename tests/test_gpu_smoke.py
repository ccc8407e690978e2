"""smoke() runs where the reference's sources, and so its library, are absent:
it needs the oracle's restatement alone."""
import pytest

pytestmark = pytest.mark.gpu


def test_smoke_without_the_reference_library(monkeypatch, capsys):
    import __graft_entry__
    from oracle import ref

    def absent():
        raise RuntimeError("the reference's library is not built")

    monkeypatch.setattr(ref, "lib", absent)
    __graft_entry__.smoke()
    assert "smoke ok" in capsys.readouterr().out
