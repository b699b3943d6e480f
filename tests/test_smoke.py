"""The smoke run of the entry points, with or without the oracle."""
import pytest


@pytest.mark.gpu
def test_smoke():
    import __graft_entry__
    __graft_entry__.smoke()
