"""Which calls of the largest grids that fit it the mesh kernel takes: short ones where
it exchanges after every step (a brush's plane leaves no room for more) stay with the
step kernels, which are faster there."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,brushes,steps,launches", [
    (1024, 1024, 0, 12, 1), (1024, 1024, 1, 12, 6), (1024, 1024, 1, 31, 16),
    (1024, 1024, 1, 32, 1), (1100, 1100, 0, 12, 6), (1100, 1100, 1, 40, 1), (960, 960, 2, 8, 1),
    (1024, 1024, 2, 40, 20)])
def test_launches(W, H, brushes, steps, launches):
    import terrainwatersim_gb300 as tws
    with tws.Grid(W, H) as g:
        g.set_sources([(tws.SOURCE_BRUSH, 300.0, 400.0 + k, 400.0, 0.01) for k in range(brushes)])
        n0 = tws.lib().tws_launch_count()
        g.step(steps)
        assert tws.lib().tws_launch_count() - n0 == launches
        g.sync()
