"""Narrow grids of many cells: the kernels chosen for them, and that the sweep and
the tiles agree there bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


# a strip of the sweep counts 112 columns, a tile 32: the sweep from 7 Mi cells (FP16
# 17 Mi) while its strips cover at most 1.4 times the tiles' columns
@pytest.mark.parametrize("W,H,flux,kind,k", [
    (16, 475000, 0, "tile", 2), (113, 67256, 0, "tile", 2), (128, 100000, 0, "tile", 2),
    (56, 135714, 0, "tile", 2), (64, 284375, 1, "tile", 2), (129, 60000, 0, "sweep", 3),
    (256, 29687, 0, "sweep", 3), (72, 105555, 0, "sweep", 3),
    (112, 67857, 0, "sweep", 3), (224, 33928, 0, "sweep", 3), (192, 94791, 1, "sweep", 3),
    (3000, 3000, 0, "sweep", 3)])
def test_sweep_where_its_strips_fit(tws, W, H, flux, kind, k):
    with tws.Grid(W, H, None, flux) as g:
        v = tws.variants()[g.current_variant()]
    assert v[0] == k
    assert v[5] == {"tile": tws.VARIANT_TILE, "sweep": tws.VARIANT_SWEEP}[kind]


@pytest.mark.parametrize("W,H,tile_y", [(8, 500000, 32), (20, 131073, 32), (256, 256, 16),
                                        (2047, 2047, 32), (2000, 2000, 16)])
def test_one_step_tile_follows_the_number_of_tiles(tws, W, H, tile_y):
    with tws.Grid(W, H) as g:
        g.set_steps_per_launch(1)
        v = tws.variants()[g.current_variant()]
    assert (v[0], v[1], v[2]) == (1, 32, tile_y)


@pytest.mark.parametrize("W", [16, 113])
def test_default_as_the_plain_kernel(tws, W):
    H = 8_000_000 // W
    out = []
    for variant in (-1, 0):
        with tws.Grid(W, H) as g:
            g.generate_scene(7, 40.0, 15.0)
            g.set_sources([(tws.SOURCE_DISK, W // 2, H // 2, 40, 0.02)])
            g.set_variant(variant)
            g.step(7)
            out.append(g.download())
    for name, x, y in zip(("depth", "flux", "flow map"), *out):
        assert_bitexact(x, y, name)


@pytest.mark.parametrize("W,H,tile_y", [(300000, 8, 16), (300000, 16, 16), (200000, 48, 16),
                                        (200000, 24, 32), (200000, 64, 32)])
def test_one_step_tile_of_flat_grids(tws, W, H, tile_y):
    """16 rows a tile where 32 would waste a third more."""
    with tws.Grid(W, H) as g:
        g.set_steps_per_launch(1)
        v = tws.variants()[g.current_variant()]
    assert (v[0], v[1], v[2]) == (1, 32, tile_y)
