"""The single-instance staged kernel's tiles, 4 rows of 32 elements
(csrc/tile.cuh, SoloTile), by the checks of the 64-column ones."""
from __future__ import annotations

import pytest

import test_tile_cover as wide


@pytest.mark.parametrize("s", [64, 65, 66, 70, 95, 96, 97, 127])
def test_tiles_cover_the_cube(monkeypatch, s):
    monkeypatch.setattr(wide, "COLS", 32)
    wide.test_tiles_cover_the_cube(s, 4)
