"""The smoke entry point leaves the process as it found it: what it asks of the
library for one run holds for no simulation made after it."""
import os

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tb2", [None, "0"])
def test_smoke_leaves_the_environment(fdtd, monkeypatch, tb2):
    import __graft_entry__ as entry

    monkeypatch.delenv("FDTDB_TB2", raising=False)
    if tb2:
        monkeypatch.setenv("FDTDB_TB2", tb2)
    before = dict(os.environ)
    entry.smoke()
    assert dict(os.environ) == before
