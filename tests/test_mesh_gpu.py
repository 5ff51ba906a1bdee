"""GPU parity of the mesh kernel (tws_mesh.cu: a grid's whole state on chip across
all SMs), which runs the long calls of grids up to about a million cells: tile
and halo edges, both borders and storages, sources, odd numbers of exchanges,
calls past one launch, grids stepped on several streams and threads at once,
and a wait limit that is not reached."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import assert_bitexact

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tws():
    import terrainwatersim_gb300 as t
    t.lib()
    return t


def state(W, H, seed):
    rng = np.random.default_rng(seed)
    b = rng.uniform(0, 6, (H, W)).astype(np.float32)
    d = np.maximum(0, rng.uniform(-2, 5, (H, W))).astype(np.float32)
    f = rng.uniform(0, 0.3, (H, W, 4)).astype(np.float32)
    return b, d, f


def reference(oracle, b, d, f, p, sources, steps, closed, scale=0.0):
    d, f = d.copy(), f.copy()
    v = np.zeros(d.shape + (2,), np.float32)
    if scale:
        oracle.quantize_f16(f, scale)
    oracle.step_f32(b.copy(), d, f, v, *p.as_tuple(),
                    oracle.BOUNDARY_CLOSED if closed else oracle.BOUNDARY_OPEN,
                    [tuple(s) for s in sources], nsteps=steps, flux_scale=scale)
    return d, f, v


def compare(got, want, what=""):
    for name, x, y in zip(("depth", "flux", "flow map"), got, want):
        assert_bitexact(x, y, f"{name} {what}")


def run(tws, oracle, W, H, steps, closed=True, flux=0, sources=(), launches=1, seed=1):
    b, d, f = state(W, H, seed)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED if closed else tws.BOUNDARY_OPEN)
    with tws.Grid(W, H, p, flux) as g:
        g.upload(b, d, f)
        g.set_sources(sources)
        n0 = tws.lib().tws_launch_count()
        g.step(steps)
        n = tws.lib().tws_launch_count() - n0
        g.sync()
        scale = g.buffers().flux_scale if flux else 0.0
        got = g.download()
    if launches is not None:
        assert n == launches
    compare(got, reference(oracle, b, d, f, p, sources, steps, closed, scale), f"{W}x{H}")


@pytest.mark.parametrize("W,H", [(1, 1), (2, 40), (7, 3), (60, 16), (61, 16), (60, 17), (64, 64),
                                 (65, 129), (128, 31), (256, 256), (333, 517), (700, 600),
                                 (1021, 763), (1024, 1024)])
@pytest.mark.parametrize("closed,flux", [(True, 0), (False, 0), (True, 1)])
def test_sizes_bitexact(tws, oracle, W, H, closed, flux):
    srcs = [(tws.SOURCE_DISK, W // 3, H // 2, min(W, H) // 5, 0.05)]
    run(tws, oracle, W, H, 13, closed, flux, srcs)


@pytest.mark.parametrize("steps", [8, 9, 10, 11, 12, 16, 17, 33])
def test_every_number_of_exchanges(tws, oracle, steps):
    run(tws, oracle, 190, 140, steps, seed=steps)


def test_sources(tws, oracle):
    """Disks and up to two brushes in any order; with a third brush the step
    kernels run.  A brush that drains below zero gives negative outflows and
    NaNs, where the oracle's FP16 mode and NaN bits differ from every packed
    kernel's: those calls are compared with the two-step tiles."""
    disk = [(tws.SOURCE_DISK, 100, 90, 40, 0.02), (tws.SOURCE_DISK, 110, 80, 30, 0.013)]
    brush = [(tws.SOURCE_BRUSH, 120.5, 60.25, 900.0, 0.3), (tws.SOURCE_BRUSH, 5.0, 2.0, 200.0, 0.5),
             (tws.SOURCE_BRUSH, 90.0, 90.0, 50.0, -0.1)]
    run(tws, oracle, 210, 150, 20, True, 0, [brush[0], disk[0], brush[1], disk[1]])
    b, d, f = state(210, 150, 1)
    for flux, srcs, launches in ((1, [disk[0], brush[2], disk[1]], 1), (0, brush + disk, 10)):
        out = []
        for variant in (-1, 16):
            with tws.Grid(210, 150, tws.params_physical(boundary=tws.BOUNDARY_OPEN), flux) as g:
                g.upload(b, d, f)
                g.set_sources(srcs)
                g.set_variant(variant)
                n0 = tws.lib().tws_launch_count()
                g.step(20)
                n = tws.lib().tws_launch_count() - n0
                out.append(g.download())
            assert n == (launches if variant == -1 else 10)
        compare(out[0], out[1])


def test_long_call_and_continued_state(tws, oracle):
    """More steps than one launch takes, then short and long calls in turn."""
    W, H = 97, 70
    b, d, f = state(W, H, 3)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    with tws.Grid(W, H, p) as g:
        g.upload(b, d, f)
        n0 = tws.lib().tws_launch_count()
        g.step(4100)
        assert tws.lib().tws_launch_count() - n0 >= 2
        for n in (3, 40, 1, 8):
            g.step(n)
        got = g.download()
    compare(got, reference(oracle, b, d, f, p, [], 4152, True))


def test_streams_and_threads(tws, oracle):
    """Grids on streams of their own, stepped from four threads at once."""
    sizes = [(256, 200), (500, 410), (90, 700), (640, 480)]
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    data = [state(W, H, 10 + i) for i, (W, H) in enumerate(sizes)]
    got = [None] * 4

    def work(i):
        W, H = sizes[i]
        with tws.Grid(W, H, p) as g:
            g.upload(*data[i])
            for _ in range(5):
                g.step(20)
            g.sync()
            got[i] = g.download()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(4):
        compare(got[i], reference(oracle, *data[i], p, [], 100, True), str(sizes[i]))


def test_depths_outside_the_packed_division(tws, oracle):
    W, H = 130, 70
    rng = np.random.default_rng(3)
    b = (rng.uniform(0, 1, (H, W)) * 10.0 ** rng.integers(-30, 8, (H, W))).astype(np.float32)
    mag = rng.choice([0.0, 1e-44, 1e-38, 1e-32, 7.8e-31, 8.0e-31, 1e-20, 1e-6, 1.0, 1e6, 1e9], (H, W))
    d = (rng.uniform(0.5, 1, (H, W)) * mag).astype(np.float32)
    f = (rng.uniform(0, 1, (H, W, 4)) * 10.0 ** rng.integers(-40, 9, (H, W, 4))).astype(np.float32)
    p = tws.params_physical(boundary=tws.BOUNDARY_CLOSED)
    with tws.Grid(W, H, p) as g:
        g.upload(b, d, f)
        g.step(8)
        got = g.download()
    compare(got, reference(oracle, b, d, f, p, [], 8, True))


def test_non_finite_cells_as_the_plain_kernel(tws):
    W, H = 300, 90
    b, d, f = state(W, H, 5)
    b[20, 30], b[40, 200], d[60, 127], d[10, 250] = np.inf, np.nan, np.inf, np.nan
    d[70, 60], f[30, 112, 1], f[50, 113, 0] = -1.0, np.inf, np.nan
    b[5, 5] = -0.0
    d[6:9, 5:9] = -0.0
    p = tws.params_physical(boundary=tws.BOUNDARY_OPEN)
    out = []
    for variant in (0, -1):
        with tws.Grid(W, H, p) as g:
            g.upload(b, d, f)
            g.set_variant(variant)
            g.step(8)
            out.append(g.download())
    for x, y in zip(out[1], out[0]):
        nan = np.isnan(y)
        assert np.array_equal(nan, np.isnan(x))
        assert np.array_equal(x[~nan].view(np.uint32), y[~nan].view(np.uint32))


def test_pinned_choices_keep_their_kernels(tws):
    """A variant, a steps-per-launch setting and the resident kernel are not
    replaced, and short calls stay with the step kernels."""
    with tws.Grid(128, 128) as g:
        def launches(n):
            n0 = tws.lib().tws_launch_count()
            g.step(n)
            return tws.lib().tws_launch_count() - n0
        assert launches(20) == 1 and launches(3) == 2
        g.set_variant(0)
        assert launches(20) == 20
        g.set_variant(-1)
        g.set_steps_per_launch(2)
        assert launches(20) == 10
        g.set_steps_per_launch(0)
        assert launches(20) == 1
        g.sync()
