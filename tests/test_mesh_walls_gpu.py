"""Closed walls where a mesh-kernel tile's box ends on them: grids as high as a
box of the kernel (16 rows of warps, RY rows each), which have no halo rows, and
wide enough for CTAs whose columns lie inside the grid.  One width for each RY
the kernel is built for, from the widths on which it takes that height whole."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

# (W, H): H = 16 * RY for RY = 1, 2, 3, 4, 5, 7 and 9; 96 and 128 have one inner tile
SIZES = [(96, 16), (128, 16), (1000, 16), (256, 32), (3000, 48), (4001, 64), (4600, 80),
         (4600, 112), (4700, 144)]


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


def state(W, H):
    rng = np.random.default_rng(H)
    b = rng.uniform(0, 6, (H, W)).astype(np.float32)
    d = rng.uniform(1, 5, (H, W)).astype(np.float32)
    f = rng.uniform(0, 0.3, (H, W, 4)).astype(np.float32)
    return b, d, f


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("closed,flux", [(True, 0), (True, 1), (False, 0)])
def test_bitexact(tws, oracle, W, H, closed, flux):
    b, d, f = state(W, H)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED if closed else tws.BOUNDARY_OPEN)
    with tws.Grid(W, H, p, flux) as g:
        g.upload(b, d, f)
        n0 = tws.lib().tws_launch_count()
        g.step(13)
        assert tws.lib().tws_launch_count() - n0 == 1  # the mesh kernel
        scale = g.buffers().flux_scale if flux else 0.0
        got = g.download()
    v = np.zeros((H, W, 2), np.float32)
    if flux:
        oracle.quantize_f16(f, scale)
    oracle.step_f32(b, d, f, v, *p.as_tuple(),
                    oracle.BOUNDARY_CLOSED if closed else oracle.BOUNDARY_OPEN, [], nsteps=13,
                    flux_scale=scale)
    for name, x, y in zip(("depth", "flux", "flow map"), got, (d, f, v)):
        assert_bitexact(x, y, name)


@pytest.mark.parametrize("W,H", SIZES)
def test_volume_stays(tws, W, H):
    """Without sources a closed grid keeps its water: each step rounds a depth (below
    16 m) to 2^-20 m at worst, each cell and step its own way."""
    b, d, f = state(W, H)
    f[:] = 0
    steps = 40
    with tws.Grid(W, H, tws.params_physical(boundary=tws.BOUNDARY_CLOSED)) as g:
        g.upload(b, d, f)
        v0 = g.volume()
        g.step(steps)
        v1 = g.volume()
    assert abs(v1 - v0) <= steps * W * H * 2.0 ** -20
