"""Who holds the mesh kernel's workspace: grids that may step by themselves, and not
those of the serving loop, whose memory budget does not count it."""
from __future__ import annotations

import gc
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    gc.collect()  # grids that earlier tests left behind
    return t


def held(tws):
    return tws.lib().tws_test_mesh_workspace()


def test_goes_with_the_last_grid(tws):
    assert held(tws) == 0
    with tws.Grid(64, 64):
        small = held(tws)
        assert small > 0
        with tws.Grid(1024, 1024):
            large = held(tws)
            assert small < large <= 64 << 20
        assert held(tws) == large
        with tws.Grid(2048, 1024):  # too large for the kernel
            assert held(tws) == large
    assert held(tws) == 0
    with tws.Grid(2048, 1024):
        assert held(tws) == 0


def requests(tws, serve, n, steps):
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    return [serve.make_request(i, 500, 400, 3 + i, 12.0, p, [], steps, 0.0) for i in range(n)]


@pytest.mark.parametrize("serial", [False, True])
def test_served_grids_do_without(tws, serial):
    from terrainwatersim_gb300 import serve
    with serve.Server(memory_budget_bytes=4e9, flux_storage=0) as srv:
        for r in requests(tws, serve, 6, 20000):
            srv.submit(r)
        srv.close_submissions()
        t = threading.Thread(target=srv.run, kwargs={"serial": serial})
        most = polls = 0
        t.start()
        while t.is_alive():
            most = max(most, held(tws))
            polls += 1
        t.join()
        assert polls > 10 and most == 0
        assert all(r.status == 0 for r in srv.results())


@pytest.mark.parametrize("serial", [False, True])
def test_kept_grids_take_it(tws, serial):
    """A grid that the loop hands on runs the mesh kernel when its owner steps it."""
    from terrainwatersim_gb300 import serve
    with serve.Server(memory_budget_bytes=4e9, flux_storage=0, keep_grids=True) as srv:
        for r in requests(tws, serve, 2, 20):
            srv.submit(r)
        srv.close_submissions()
        srv.run(serial=serial)
        for res in srv.results():
            g = res.grid
            L = tws.lib()
            assert L.tws_set_variant(g._h, -1) == 0
            n0 = L.tws_launch_count()
            assert L.tws_step(g._h, 40) == 0
            assert L.tws_launch_count() - n0 == 1
            assert L.tws_sync(g._h) == 0
            g.close()
    assert held(tws) == 0
