"""The autotuner and the mesh kernel: what a tuned grid and later grids of its shape
run.  Each test has a shape of its own (choices are kept for the process)."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


def launches(tws, g, steps):
    n0 = tws.lib().tws_launch_count()
    g.step(steps)
    g.sync()
    return tws.lib().tws_launch_count() - n0


def scene(tws, W, H, **kw):
    g = tws.Grid(W, H, **kw)
    g.generate_scene(1, 40.0, 15.0)
    return g


def test_tuning_where_the_mesh_kernel_cannot_run_does_not_rule_it_out(tws):
    W, H = 640, 400  # more than the resident kernel takes
    with scene(tws, W, H) as g:
        g.set_sources([(tws.SOURCE_BRUSH, 20.0 * k, 30.0, 50.0, 0.1) for k in range(3)])
        best = g.autotune(24)
        assert 0 <= best < len(tws.variants())
        assert launches(tws, g, 40) > 1
    with scene(tws, W, H) as g:
        assert launches(tws, g, 40) == 1
