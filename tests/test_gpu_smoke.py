"""The smoke entry point of the repository runs to its end on the GPU (its lattice is a plane
one, whose moment loop takes several Chebyshev steps per launch)."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_smoke_entry_point(capsys):
    import __graft_entry__

    __graft_entry__.smoke()
    assert "smoke ok" in capsys.readouterr().out
