"""Small grids on streams of their own: none waits for another's stream.  One
stream is held up by a kernel that sleeps for a while; what the others do
meanwhile must be done before it wakes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu

SLEEP = 1_000_000_000  # SM clocks, about half a second


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


@pytest.fixture()
def held(tws):
    """A stream with a 128 x 128 grid whose 40 steps wait behind a sleeping kernel;
    yields (grid, state, done) with done() true once the steps have run."""
    import torch
    torch.cuda._sleep(1000)  # the kernel is loaded
    stream = torch.cuda.Stream()
    with tws.Grid(128, 128, params(tws), stream=stream.cuda_stream) as g:
        data = state(128, 128)
        # (a kernel's first launch loads it, which waits for the device)
        for W, H in ((128, 128), (60, 16), (700, 600)):
            with tws.Grid(W, H, params(tws)) as warm:
                warm.upload(*state(W, H))
                warm.step(24)
                warm.set_steps_per_launch(2)
                warm.step(4)
                warm.download()
        g.upload(*data)
        event = torch.cuda.Event()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(SLEEP)
        g.step(40)
        event.record(stream)
        yield g, data, event.query
        stream.synchronize()


def params(tws):
    return tws.params_physical(boundary=tws.BOUNDARY_CLOSED)


def state(W, H):
    rng = np.random.default_rng(W * H)
    b = rng.uniform(0, 6, (H, W)).astype(np.float32)
    d = np.maximum(0, rng.uniform(-2, 5, (H, W))).astype(np.float32)
    f = rng.uniform(0, 0.3, (H, W, 4)).astype(np.float32)
    return b, d, f


def check(tws, oracle, grid, data, steps):
    compare(tws, oracle, grid.download(), data, steps)


def compare(tws, oracle, got, data, steps):
    b, d, f = (a.copy() for a in data)
    v = np.zeros(d.shape + (2,), np.float32)
    oracle.step_f32(b, d, f, v, *params(tws).as_tuple(), oracle.BOUNDARY_CLOSED, [], nsteps=steps)
    for name, x, y in zip(("depth", "flux", "flow map"), got, (d, f, v)):
        assert_bitexact(x, y, name)


def launches(tws, g, steps):
    n0 = tws.lib().tws_launch_count()
    g.step(steps)
    return tws.lib().tws_launch_count() - n0


@pytest.mark.parametrize("W,H,alone", [(200, 150, False), (60, 16, True)])
def test_steps_pass_a_held_stream(tws, oracle, held, W, H, alone):
    g0, data0, done0 = held
    with tws.Grid(W, H, params(tws)) as g:
        data = state(W, H)
        g.upload(*data)
        n = launches(tws, g, 40)
        g.sync()
        assert not done0()
        assert n == (1 if alone else 20)  # (a grid of one CTA waits for no other)
        check(tws, oracle, g, data, 40)
        g0.sync()
        assert launches(tws, g, 40) == 1  # the mesh kernel again
        check(tws, oracle, g, data, 80)
    check(tws, oracle, g0, data0, 40)


def test_creating_and_destroying_passes_a_held_stream(tws, oracle, held):
    """A larger grid grows the workspace that the held launch uses, and its
    destruction gives nothing back that the launch needs."""
    g0, data0, done0 = held
    with tws.Grid(700, 600, params(tws)) as g:
        data = state(700, 600)
        g.upload(*data)
        g.step(24)
        g.sync()
        assert not done0()
        got = g.download()
    assert not done0()
    compare(tws, oracle, got, data, 24)
    check(tws, oracle, g0, data0, 40)


def test_last_grid_destroyed_with_work_queued(tws, oracle):
    """The workspace outlives the queued work of the last grid; the next grid has
    one of its own."""
    import torch
    stream = torch.cuda.Stream()
    g = tws.Grid(300, 200, params(tws), stream=stream.cuda_stream)
    data = state(300, 200)
    g.upload(*data)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(SLEEP // 4)
    g.step(400)
    g.close()
    event = torch.cuda.Event()
    event.record(stream)
    with tws.Grid(300, 200, params(tws)) as g:
        g.upload(*data)
        g.step(24)
        check(tws, oracle, g, data, 24)
    stream.synchronize()
    assert event.query()


def test_destroyed_grids_work_still_counts(tws, oracle):
    """The last grid is gone, its launch is not: a new grid's steps go beside it as
    tiles, and as the mesh kernel once it has run."""
    import torch
    stream = torch.cuda.Stream()
    for W, H in ((200, 150), (300, 200)):  # (the kernels are loaded)
        with tws.Grid(W, H, params(tws)) as warm:
            warm.step(24)
            warm.set_steps_per_launch(2)
            warm.step(4)
            warm.sync()
    g = tws.Grid(300, 200, params(tws), stream=stream.cuda_stream)
    g.upload(*state(300, 200))
    with torch.cuda.stream(stream):
        torch.cuda._sleep(SLEEP)
    g.step(400)
    g.close()
    event = torch.cuda.Event()
    event.record(stream)
    with tws.Grid(200, 150, params(tws)) as g:
        data = state(200, 150)
        g.upload(*data)
        n = launches(tws, g, 24)
        g.sync()
        assert not event.query()
        assert n == 12
        stream.synchronize()
        assert launches(tws, g, 24) == 1
        check(tws, oracle, g, data, 48)


def test_many_streams_in_turn(tws, oracle):
    """More streams than entries stay, stepped in turn without waiting."""
    import torch
    grids = [tws.Grid(96 + 8 * i, 80, params(tws), stream=torch.cuda.Stream().cuda_stream)
             for i in range(12)]
    data = [state(g.width, g.height) for g in grids]
    for g, d in zip(grids, data):
        g.upload(*d)
    for _ in range(6):
        for g in grids:
            g.step(10)
    for g, d in zip(grids, data):
        check(tws, oracle, g, d, 60)
        g.close()
