"""The package's entry point: a tiny dry and a tiny moist run on the GPU against
the oracle, with the kernel launches they take."""
import pytest

pytestmark = pytest.mark.gpu


def test_smoke(cress, oracle_lib, capsys):
    import __graft_entry__ as entry
    entry.smoke()
    assert capsys.readouterr().out.count("smoke ok") == 2
