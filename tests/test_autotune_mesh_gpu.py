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


@pytest.mark.parametrize("W,H", [(64, 48), (72, 64)])
def test_resident_is_reported_where_it_runs(tws, W, H):
    """Lost borders (the test hook) end a mesh launch; the resident kernel has no
    such wait."""
    with scene(tws, W, H) as g:
        best = g.autotune(240)
        g.set_wait_limit(2_000_000)
        g.test_drop_tile_loads(True)
        n = 0
        try:
            n = launches(tws, g, 40)
            mesh = False
        except tws.TwsError as e:
            assert e.code == tws.ERR_TIMEOUT
            mesh = True
        if best == tws.VARIANT_RESIDENT:
            assert not mesh and n == 1
        else:
            assert 0 <= best < len(tws.variants())


def test_tuning_supersedes_a_steps_per_launch_setting(tws):
    with scene(tws, 208, 176) as g:
        g.set_steps_per_launch(1)
        assert launches(tws, g, 40) == 40
        best = g.autotune(240)
        n = launches(tws, g, 40)
        if best == tws.VARIANT_RESIDENT:
            assert n == 1
        else:
            assert n in (1, 40 // tws.variants()[best][0])
            assert n < 40
