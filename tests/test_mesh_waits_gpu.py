"""The mesh kernel's bounded waits: one that runs out (the tiles send their
neighbours nothing) ends the launch with a time-out and the grid recovers, and
a sound call does not run out of time under a wait limit made for tile loads or
while another stream's kernel holds SMs that the launch needs."""
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


def params(tws):
    return tws.params_physical(boundary=tws.BOUNDARY_CLOSED)


def state(W, H):
    rng = np.random.default_rng(W + H)
    b = rng.uniform(0, 6, (H, W)).astype(np.float32)
    d = np.maximum(0, rng.uniform(-2, 5, (H, W))).astype(np.float32)
    f = rng.uniform(0, 0.3, (H, W, 4)).astype(np.float32)
    return b, d, f


def check(tws, oracle, got, data, steps):
    b, d, f = (a.copy() for a in data)
    v = np.zeros(d.shape + (2,), np.float32)
    oracle.step_f32(b, d, f, v, *params(tws).as_tuple(), oracle.BOUNDARY_CLOSED, [], nsteps=steps)
    for name, x, y in zip(("depth", "flux", "flow map"), got, (d, f, v)):
        assert_bitexact(x, y, name)


def mesh_steps(tws, g, steps):
    n0 = tws.lib().tws_launch_count()
    g.step(steps)
    assert tws.lib().tws_launch_count() - n0 == 1


@pytest.mark.parametrize("W,H", [(64, 64), (256, 200), (700, 600), (1024, 1024), (40, 400)])
def test_lost_border_times_out_and_grid_recovers(tws, oracle, W, H):
    data = state(W, H)
    with tws.Grid(W, H, params(tws)) as g:
        g.upload(*data)
        g.set_wait_limit(2_000_000)
        g.test_drop_tile_loads(True)
        mesh_steps(tws, g, 20)
        with pytest.raises(tws.TwsError) as e:
            g.sync()
        assert e.value.code == tws.ERR_TIMEOUT
        g.sync()  # reported once
        g.test_drop_tile_loads(False)
        g.set_wait_limit(0)
        g.upload(*data)
        mesh_steps(tws, g, 20)
        mesh_steps(tws, g, 17)
        g.sync()
        check(tws, oracle, g.download(), data, 37)


@pytest.mark.parametrize("W,H", [(60, 16), (33, 9), (256, 256)])
def test_hook_reaches_calls_without_an_exchange(tws, W, H):
    """A grid of one tile, and a call too short for an exchange: the step kernels
    run, whose loads can be lost."""
    with tws.Grid(W, H, params(tws)) as g:
        g.upload(*state(W, H))
        g.set_wait_limit(2_000_000)
        g.test_drop_tile_loads(True)
        g.step(4)
        with pytest.raises(tws.TwsError) as e:
            g.sync()
        assert e.value.code == tws.ERR_TIMEOUT


@pytest.mark.parametrize("limit", [1, 3000, 2 ** 63 - 1])
@pytest.mark.parametrize("W,H", [(64, 64), (256, 200), (1024, 1024)])
def test_any_wait_limit_leaves_a_sound_call(tws, oracle, W, H, limit):
    data = state(W, H)
    with tws.Grid(W, H, params(tws)) as g:
        g.upload(*data)
        g.set_wait_limit(limit)
        mesh_steps(tws, g, 40)
        g.sync()
        check(tws, oracle, g.download(), data, 40)


def test_waits_for_sms_do_not_count(tws, oracle):
    """A resident grid holds 16 SMs for tens of milliseconds; a mesh launch that
    needs all SMs, queued meanwhile, waits for them longer than its limit."""
    data = state(1024, 1024)
    with tws.Grid(256, 256, params(tws)) as r, tws.Grid(1024, 1024, params(tws)) as g:
        r.upload(*state(256, 256))
        r.set_resident(16)
        r.step(8)
        g.upload(*data)
        mesh_steps(tws, g, 16)
        g.upload(*data)
        g.set_wait_limit(1)
        r.step(4096 * 4)
        mesh_steps(tws, g, 16)
        g.sync()
        r.sync()
        check(tws, oracle, g.download(), data, 16)
