"""Where a launch of the mesh kernel is refused, the step kernels run the call."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,flux", [(256, 200, 0), (60, 16, 0), (130, 97, 1)])
def test_refused_launch_runs_as_tiles(oracle, W, H, flux):
    import terrainwatersim_gb300 as tws
    rng = np.random.default_rng(5)
    b = rng.uniform(0, 6, (H, W)).astype(np.float32)
    d = np.maximum(0, rng.uniform(-2, 5, (H, W))).astype(np.float32)
    f = np.zeros((H, W, 4), np.float32)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)

    def launches(g, n):
        n0 = tws.lib().tws_launch_count()
        g.step(n)
        return tws.lib().tws_launch_count() - n0

    with tws.Grid(W, H, p, flux) as g:
        g.upload(b, d, f)
        assert launches(g, 20) == 1
        g.test_refuse_mesh(True)
        assert launches(g, 21) > 10
        g.sync()
        g.test_refuse_mesh(False)
        assert launches(g, 20) == 1
        scale = g.buffers().flux_scale if flux else 0.0
        got = g.download()
        for bad in (-1, 2):
            assert tws.lib().tws_test_refuse_mesh(g._h, bad) == tws.ERR_INVALID
    v = np.zeros((H, W, 2), np.float32)
    oracle.step_f32(b, d, f, v, *p.as_tuple(), oracle.BOUNDARY_CLOSED, [], nsteps=61,
                    flux_scale=scale)
    for name, x, y in zip(("depth", "flux", "flow map"), got, (d, f, v)):
        assert_bitexact(x, y, name)
