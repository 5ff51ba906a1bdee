"""tws_grid_bytes, by which the serving loop admits, counts all that a grid
allocates (a CPU test: the entry point is host-only)."""
from __future__ import annotations

import pytest


@pytest.mark.parametrize("W,H", [(1, 1), (64, 64), (97, 70), (1024, 1024), (16384, 16384)])
@pytest.mark.parametrize("flux,flux_bytes", [(0, 16), (1, 8)])
def test_counts_state_and_scratch(W, H, flux, flux_bytes):
    from terrainwatersim_gb300 import build
    build.build()
    import terrainwatersim_gb300 as tws
    cells = (W + 31) // 32 * 32 * H
    state = cells * (4 + 2 * 4 + 2 * flux_bytes + 8)  # terrain, two depths, two fluxes, flow map
    scratch = 8 * 4096  # the row sweep's ranges: a word for each resident warp
    maps = 5 * 128 * len(tws.variants())
    got = tws.lib().tws_grid_bytes(W, H, flux)
    least = state + scratch + maps
    # besides: the sums of tws_volume, the error word, and parts on 256-byte boundaries
    assert least < got <= least + 32768
    assert got % 256 == 0
    assert tws.lib().tws_grid_bytes(0, H, flux) == 0
