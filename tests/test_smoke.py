"""The smoke run goes through every route of the lazy joins (it raises where one
launches other kernels than that route's)."""
import pytest

import __graft_entry__

pytestmark = pytest.mark.gpu


def test_smoke(capsys):
    __graft_entry__.smoke()
    out = capsys.readouterr().out
    for route in ("one launch", "one pass, chained", "two passes, chained", "one pass, sorted", "two passes, sorted",
                  "NPO table", "two passes, hashed", "batched windows"):
        assert f"smoke ok: {route}" in out
